"""Timed cases of the library's public entry points, over the sizes its users run.

The library searches the neighbourhood of powers-of-two Turing machines, sizes
such searches, runs whole tables, and checks survivors.  Each case is one call
(or one serve session) through the ctypes binding, as a program that keeps one
device context makes it.  Inputs come from the seed: it picks the deleted
state, the base machine, the share of a search or the survivors, and relabels
the states other than the start state, which changes the tables and the order
of the work but not its size.

Outputs are whole numbers (and, for the size estimate, doubles that are sums
of whole weights), so every output has one right value.
"""
import ctypes
import gzip
import math
import os
import random
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "erdos-machine-13_b200"))

import e13b200 as E  # noqa: E402

GOLD = os.path.join(ROOT, "tests", "golden")
OPS_PER_STEP = 16  # integer operations of one simulated step of the filter

# Deleted states by the size of their search, so that every seed gives a search
# of the same order: (states, mean leaves, mean simulated steps) by changed cells.
SMALL, LARGE = (2, 3, 4, 9, 10, 12, 13), (0, 1, 5, 6, 7, 8, 11)
EDITS = {
    (2, "small"): (SMALL, 1.02e3, 1.52e5), (2, "large"): (LARGE, 2.04e4, 3.14e6),
    (3, "small"): (SMALL, 4.22e5, 5.62e7), (3, "large"): (LARGE, 4.78e6, 5.16e8),
    (4, "small"): (SMALL, 9.97e7, 9.8e9), (4, "large"): (LARGE, 7.55e8, 7.4e10),
}
ALL_EDITS = {2: (1.50e5, 2.30e7), 3: (3.64e7, 4.00e9), 4: (5.99e9, 5.86e11)}  # every state: leaves, steps
CHECKED = ["check/counter_plus_f2.txt", "check/counter_plus_f3.txt", "check/f4_unread.txt"]  # lines to check again
COUNTER_FREE = ["D0", "G0", "K0", "K1", "L1", "M1"]
MOST_SURVIVORS, MOST_TEXT = 256, 8192  # rows of a survivor table, bytes of one survivor's verdicts
NODE_BYTES, RECORD_BYTES = 320, 160  # one frontier node, one survivor record


def listed():
    return [
        # one local-edit search of a small family: the shortest search a user starts
        {"name": "edits2_small", "kind": "search", "edits": 2, "size": "small"},
        # a counter machine's 2-edit neighbourhood: one of the 61 searches of that study
        {"name": "counter_neighbours", "kind": "neighbours", "edits": 2},
        # one deleted state with up to 3 changed cells: the everyday search
        {"name": "edits3_large", "kind": "search", "edits": 3, "size": "large"},
        # the same with up to 4 changed cells: a search of 5e7 to 1e8 machines
        {"name": "edits4_small", "kind": "search", "edits": 4, "size": "small"},
        # the counter search with relabel symmetry: 3.08e9 machines, the largest single search
        {"name": "counter_symmetric", "kind": "counter"},
        # all 14 deleted states at 3 changed cells, together in one serve session
        {"name": "serve_edits3", "kind": "serve", "edits": 3, "shards": 1},
        # one GPU's quarter of the 14 searches at 4 changed cells
        {"name": "serve_edits4_quarter", "kind": "serve", "edits": 4, "shards": 4},
        # sizing a search before it is started
        {"name": "estimate_4096", "kind": "estimate", "edits": 3, "size": "large", "probes": 4096},
        # a million random tables without the filter
        {"name": "raw_million", "kind": "raw", "machines": 1000000, "states": 13, "max_steps": 1 << 18},
        # whole mutant tables from the blank tape
        {"name": "tables_20000", "kind": "tables", "machines": 20000, "edits": 2},
        # the deep check behind a search: its 61 survivors to stage 12
        {"name": "recheck_61", "kind": "check", "mode": "recheck", "survivors": 61, "stages": 12},
        # stages and crafted starts of a few survivors, with their text
        {"name": "crafted_8", "kind": "crafted", "survivors": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "neighbours", "serve", "estimate", "raw", "tables", "check", "crafted"])
    if kind == "search":
        return {"kind": kind, "edits": rng.randint(2, 4), "size": rng.choice(["small", "large"]),
                "block": rng.choice([768, 768, 512, 96])}
    if kind == "neighbours":
        return {"kind": kind, "edits": rng.randint(1, 2), "slice": rng.choice([24, 24, 8, 33])}
    if kind == "serve":
        edits = rng.randint(2, 4)
        return {"kind": kind, "edits": edits, "shards": rng.randint(4, 24) if edits == 4 else rng.randint(1, 9)}
    if kind == "estimate":
        return {"kind": kind, "edits": rng.randint(2, 4), "size": rng.choice(["small", "large"]),
                "probes": _log_int(rng, 64, 20000)}
    if kind == "raw":
        return {"kind": kind, "machines": _log_int(rng, 500, 1000000), "states": rng.randint(2, 16),
                "max_steps": _log_int(rng, 1000, 1 << 18)}
    if kind == "tables":
        return {"kind": kind, "machines": _log_int(rng, 100, 100000), "edits": rng.randint(1, 3)}
    if kind == "check":
        return {"kind": kind, "mode": rng.choice(["recheck", "deep"]), "survivors": _log_int(rng, 1, 1000),
                "stages": rng.randint(8, 12)}
    return {"kind": kind, "survivors": rng.randint(1, 40)}


_context = None


def context():
    """The process's device context: a program makes one and keeps it."""
    global _context
    if _context is None:
        _context = E.Context(0)
    return _context


def machine(name):
    return E.load_machine(os.path.join(GOLD, "machines", name))


def relabelled(base, seed, keep=()):
    """base with its states renamed at random (not the start state, not those
    in keep); returns the table and the new name of every state."""
    n = len(base) // 2
    moved = [q for q in range(1, n) if q not in keep]
    to = moved[:]
    random.Random(seed).shuffle(to)
    name = list(range(n))
    for a, b in zip(moved, to):
        name[a] = b
    out = [E.E13_HALT] * (2 * n)
    for q in range(n):
        for s in (0, 1):
            c = base[2 * q + s]
            out[2 * name[q] + s] = c if c < 0 else (name[c >> 2] << 2) | (c & 3)
    return out, name


def survivor_lines(name):
    path = os.path.join(GOLD, name)
    opened = gzip.open if name.endswith(".gz") else open
    with opened(path, "rt") as f:
        return [line.rstrip("\n") for line in f if line.strip()]


def edit_job(case, seed):
    states = EDITS[case["edits"], case["size"]][0]
    base, name = relabelled(machine("erdos_14.txt"), seed)
    _, job = E.setup(base, name[states[seed % len(states)]], fmax=case["edits"])
    return job


def prepare(case, seed):
    kind, rng = case["kind"], random.Random(seed)
    state = {"kind": kind, "ctx": context()}
    if kind == "search":
        state["job"] = edit_job(case, seed)
        state["tune"] = E.tuning(block=case["block"]) if "block" in case else None
    elif kind == "neighbours":
        base, _ = relabelled(machine("counters_3state/base_%02d.txt" % (1 + seed % 61)), seed)
        state["job"] = E.setup(base, -1, fmax=case["edits"])[1]
        state["tune"] = E.tuning(slice=case["slice"]) if "slice" in case else None
    elif kind == "counter":
        base, name = relabelled(machine("erdos_14.txt"), seed, keep=(10, 11, 12, 13))
        free = [chr(65 + name[ord(c[0]) - 65]) + c[1] for c in COUNTER_FREE]
        state["job"] = E.setup(base, 13, free_cells=free, lo=10, hi=13)[1]
        state["tune"] = None
    elif kind == "serve":
        base, _ = relabelled(machine("erdos_14.txt"), seed)
        jobs = (E.setup(base, X, fmax=case["edits"]) for X in range(14))
        state["jobs"] = [job for r, job in jobs if r == 0]
        state["shard"], state["shards"] = seed % case["shards"], case["shards"]
        state["tune"] = E.tuning(epoch_us=200000)
    elif kind == "estimate":
        state["job"], state["probes"], state["seed"] = edit_job(case, seed), case["probes"], seed & 0xFFFF
    elif kind == "raw":
        state.update(n=case["machines"], nq=case["states"], max_steps=case["max_steps"], seed=seed)
    elif kind == "tables":
        base, _ = relabelled(machine("erdos_14.txt"), seed)
        gen = np.random.default_rng(seed)
        n, cells = case["machines"], len(base)
        tabs = np.full((n, E.E13_MAXCELLS), E.E13_HALT, np.int32)
        tabs[:, :cells] = base
        for _ in range(case["edits"]):
            tabs[np.arange(n), gen.integers(0, cells, n)] = gen.integers(-1, 2 * cells, n)
        state.update(n=n, nq=cells // 2, tabs=tabs)
    elif kind == "check":
        lines = survivor_lines("surv/counter_sym.txt")
        if case["survivors"] > len(lines):
            lines = survivor_lines("surv/division_v1_1RD.txt.gz")
        lines = rng.sample(lines, case["survivors"])
        state["ins"] = [E.parse_survivor_line(line) for line in lines]
        state["nmax"], state["mode"] = case["stages"], 1 if case["mode"] == "deep" else 0
    else:
        lines = [line for name in CHECKED for line in survivor_lines(name) if "table=" in line]
        state["lines"] = rng.sample(lines, case["survivors"])
    return state


def records(survivors):
    """Survivor records as sorted rows (their order is not part of the result),
    in a table of a fixed size, as the counts of two seeds differ."""
    rows = [list(s.tab) + [s.read_mask, s.st0, s.head0, s.abs_ok, s.rel_ok, s.steps] for s in survivors]
    out = np.zeros((max(MOST_SURVIVORS, len(rows)), E.E13_MAXCELLS + 6), np.int64)
    if rows:
        out[: len(rows)] = sorted(rows)
    return out


def totals(c):
    return np.array([c.leaves, c.survivors, c.steps] + list(c.hist), np.uint64).view(np.int64)


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind in ("search", "neighbours", "counter"):
        counts, survivors = ctx.search(state["job"], state["tune"])
        return {"counts": totals(counts), "survivors": records(survivors)}
    if kind == "serve":
        with E.Server(ctx, state["tune"]) as server:
            done = server.run_all(state["jobs"], shard=state["shard"], nshards=state["shards"])
        return {"counts": np.stack([totals(done[i][0].counts) for i in sorted(done)]),
                "survivors": [records(done[i][1]) for i in sorted(done)]}
    if kind == "estimate":
        out, _ = ctx.estimate(state["job"], state["probes"], state["seed"])
        return {"mean": np.array(out.mean), "std_error": np.array(out.std_error)}
    if kind == "raw":
        rows, steps = ctx.raw_run(state["n"], nq=state["nq"], max_steps=state["max_steps"], seed=state["seed"],
                                  as_array=True)
        return {"rows": np.frombuffer(rows, np.int64).reshape(-1, 4), "steps": steps}
    if kind == "tables":
        out = np.empty((state["n"], 7), np.int64)
        r = E.lib().e13_run_full(ctx.h, state["tabs"].ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), state["n"],
                                 state["nq"], out.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)))
        if r:
            raise E.E13Error(r, "e13_run_full")
        return out
    if kind == "check":
        outs = ctx.check(state["ins"], state["nmax"], state["mode"])
        return np.frombuffer(b"".join(bytes(o) for o in outs), np.int32).reshape(len(outs), -1)
    text = "\n".join(ctx.check_crafted(state["lines"])).encode()
    return np.frombuffer(text.ljust(MOST_TEXT * len(state["lines"]), b" "), np.uint8)


def exact(case, seed):
    """Whole numbers need no other value; the estimate's doubles come from
    millions of simulated steps, minutes in plain Python."""
    return None


def work(case):
    """What one pass cannot do without: its inputs and outputs, and the integer
    operations of its simulated steps (means over the seeds; the deep check and
    the crafted starts by the steps their machines take to the last stage)."""
    kind = case["kind"]
    node = NODE_BYTES + 8 * 13
    if kind == "search":
        return {"bytes": node, "flops": OPS_PER_STEP * EDITS[case["edits"], case["size"]][2]}
    if kind == "neighbours":
        return {"bytes": node + 20 * RECORD_BYTES, "flops": OPS_PER_STEP * {1: 1.5e6, 2: 1.3e8}[case["edits"]]}
    if kind == "counter":
        return {"bytes": node + 61 * RECORD_BYTES, "flops": OPS_PER_STEP * 3.19e11}
    if kind == "serve":
        return {"bytes": 14 * node, "flops": OPS_PER_STEP * ALL_EDITS[case["edits"]][1] / case["shards"]}
    if kind == "estimate":
        return {"bytes": NODE_BYTES + 32 * case["probes"], "flops": OPS_PER_STEP * 1e4 * case["probes"]}
    if kind == "raw":
        # about one random machine in ten runs to the limit, the others leave the window or halt early
        return {"bytes": 32 * case["machines"],
                "flops": OPS_PER_STEP * case["machines"] * (1000 + 0.11 * case["max_steps"])}
    if kind == "tables":
        return {"bytes": case["machines"] * (4 * E.E13_MAXCELLS + 56), "flops": OPS_PER_STEP * 1.2e4 * case["machines"]}
    if kind == "check":
        return {"bytes": case["survivors"] * (ctypes.sizeof(E.CheckIn) + ctypes.sizeof(E.CheckOut)),
                "flops": OPS_PER_STEP * 0.8 * 4.0 ** case["stages"] * case["survivors"]}
    return {"bytes": 1000 * case["survivors"], "flops": OPS_PER_STEP * 3.5e6 * 3 * case["survivors"]}
