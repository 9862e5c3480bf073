"""e13_tuning::epoch_us bounds an epoch of a serve session: the search kernel and
the long-machine kernel behind it together."""
import statistics

import pytest

import e13b200 as E
from gpu_common import ctx, make_job

pytestmark = pytest.mark.gpu


def test_epochs_keep_their_bound(searches):
    """Epochs of 5 ms of a search that always has long machines unfinished at
    their end, so that both kernels use all of their time.  Dealing out and
    collecting the frontier's 10^5 nodes of 320 bytes takes some 0.2 ms more;
    0.6 ms leaves room for it, and none for 1 ms of the second kernel."""
    with E.Server(ctx(), E.tuning(epoch_us=5000)) as srv:
        srv.submit(make_job(searches["local_edits_f4"], 8), 0)
        ms = [0.0]
        for _ in range(14):
            srv.step()
            ms.append(srv.stats()[0])
    assert statistics.median(b - a for a, b in list(zip(ms, ms[1:]))[2:]) < 5.6


def test_epochs_with_many_long_machines_keep_their_bound(searches):
    """Epochs of 20 ms of the same search, which gathers long machines: from the
    sixth on thousands of them are unfinished at the end of each epoch.  Beside
    the 0.2 ms above an epoch may wait for a survivor's read mask (a run of
    some 271,500 steps by visits, below 1 ms); 22 ms holds both, and not the
    4 to 8 ms that handing out so many machines one by one took.  (One epoch may
    be longer: a survivor found by the search kernel itself is run step by step.)"""
    with E.Server(ctx(), E.tuning(epoch_us=20000)) as srv:
        srv.submit(make_job(searches["local_edits_f4"], 8), 0)
        ms = [0.0]
        for _ in range(14):
            srv.step()
            ms.append(srv.stats()[0])
    assert sorted(b - a for a, b in zip(ms, ms[1:]))[-2] < 22
