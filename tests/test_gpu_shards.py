"""Many shares of one job: each call expands the job again, so they add up only if
every expansion leaves the same frontier, with long machines of the job stopped
at the same steps."""
import pytest

import e13b200 as E
from gpu_common import check_entry, ctx, golden_lines, make_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,nshards", [(8, 24), (8, 64), (12, 48)])
def test_many_shards_add_up_to_the_search(searches, X, nshards):
    """Leaves, steps, deaths by stage and survivor lines of all shards are the
    search's, with shards run under different tunings, as their ranks may."""
    e = searches["local_edits_f3"]
    job = make_job(e, X)
    tunes = [E.tuning(), E.tuning(block=96), E.tuning(kernel=0, block=256, step_cap=300), E.tuning(slice=7)]
    total = dict(leaves=0, survivors=0, steps=0, hist=[0] * 10)
    lines = []
    for shard in range(nshards):
        counts, surv = ctx().search_shard(job, shard, nshards, tunes[shard % len(tunes)])
        c = counts.as_dict()
        for k in ("leaves", "survivors", "steps"):
            total[k] += c[k]
        total["hist"] = [a + b for a, b in zip(total["hist"], c["hist"])]
        lines += [E.survivor_line(job, s) for s in surv]
    check_entry(dict(e, expect=[x for x in e["expect"] if x["X"] == X]), [total])
    assert sorted(lines) == [l for l in golden_lines(e) if f" X={X} " in l]


@pytest.mark.parametrize("X", [8, 10])
def test_a_share_is_the_same_in_every_call(searches, X):
    job = make_job(searches["local_edits_f3"], X)
    for shard in (0, 17):
        got = [ctx().search_shard(job, shard, 40, E.tuning(block=b))[0].as_dict() for b in (768, 768, 64, 512)]
        assert all(g == got[0] for g in got)
