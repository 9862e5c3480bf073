"""What a context keeps between calls does not keep a later call from memory:
a serve session's second stack and the calls' working memory are given back
when a buffer of the context finds no room without them."""
import pytest
import torch

import e13b200 as E
from gpu_common import check_entry, make_job

pytestmark = pytest.mark.gpu

NODE = 320


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def search(c, e, X, **tune):
    counts, _ = c.search(make_job(e, X), E.tuning(**tune))
    check_entry(dict(e, expect=[x for x in e["expect"] if x["X"] == X]), [counts.as_dict()])


def test_a_large_session_leaves_room_for_a_larger_search(searches):
    """A session's two stacks hold four fifths of the memory; a search on the
    same context may then have a stack of seven tenths."""
    e = searches["local_edits_f2"]
    nodes = free_bytes() // NODE
    with E.Context(0) as c:
        with E.Server(c, E.tuning(stack_nodes=int(0.4 * nodes))) as srv:
            got = srv.run_all([make_job(e, 3)])
            assert got[0][0].status == 0
        search(c, e, 3, stack_nodes=int(0.7 * nodes))


def test_a_default_session_leaves_room_for_the_largest_search(searches):
    """The default session's second stack (5.4 GB) is kept for the next session,
    until a search needs more than what else is free."""
    e = searches["local_edits_f2"]
    with E.Context(0) as c:
        for _ in range(2):
            with E.Server(c) as srv:
                assert srv.run_all([make_job(e, 3)])[0][0].status == 0
        kept = 16 << 20
        search(c, e, 3, stack_nodes=free_bytes() // NODE + kept + kept // 2)


def test_working_memory_leaves_room_for_a_search(searches):
    """A recheck's tapes (1 MB a machine, kept up to 1 GB) go when a search needs them."""
    e = searches["local_edits_f2"]
    line = ("SURVIVOR X=9 st0=2 head0=-2 abs=1 rel=0 steps=271500 table=1L1 1R0|1L2 1L1|1R3 0R0|0L6 0R4|0L3 1R5|0R1 1R4|"
            "1R3 1L7|1L6 0L8|1L3 0L7|?0L10 ?1R9|?1R12 ?0L2|?0L12 ?---|?0R9 ?0L11")
    with E.Context(0) as c:
        search(c, e, 3)
        before = free_bytes()
        c.check([E.parse_survivor_line(line)] * 1000, 4, 0)
        kept = before - free_bytes()
        assert kept > 900 << 20
        own = 4 << 20  # the stack the context has: freed before the larger one is asked for
        search(c, e, 3, stack_nodes=free_bytes() // NODE + own + (kept // 2) // NODE)


def test_raw_machines_run_without_room_for_their_list():
    """Totals of machines generated on the device need no memory by their number:
    where the list of the ones that live long (4 bytes a machine, for a limit
    that makes it worth while) finds no room, they run all the same."""
    n, most = 1 << 24, 12000
    with E.Context(0) as c:
        c.raw_run(1000, max_steps=most, want_out=False)
        held = torch.empty(free_bytes() - (32 << 20), dtype=torch.uint8, device="cuda")
        try:
            _, without = c.raw_run(n, max_steps=most, want_out=False)
        finally:
            del held
            torch.cuda.empty_cache()
        _, total = c.raw_run(n, max_steps=most, want_out=False)
    assert without == total
