"""Performance cases: what a program that uses this framework has it do.

A case is a dict of plain values.  `listed()` names the standing ones, `draw(rng)` gives another of the same
ranges, `prepare` makes what a program holds before the call (graph, table, buffers), `run` is one pass through
the public entry points, `work` is what a pass cannot do without, `tolerance` how far outputs may be apart.

Graphs are seeded and synthetic, made on the GPU by the framework's own generators: directed or undirected R-MAT
and a capped power-law graph, with weights uniform in [1, 10) as the generators leave them or log-normal ones
(few heavy edges, many light ones).  A case's graph has one structure; weights, start vertices and draws come
from the seed.  Walks and trees are keyed by counters, tables are integer constructions, so
every output is compared exactly.
"""
import math

import numpy as np
import torch

from skywalker_b200 import (APP_DEEPWALK, APP_NODE2VEC, APP_PPR, KHOP_DISTINCT, KHOP_TAKE_ALL, KHOP_UNBIASED,
                            MODE_OFFLINE, MODE_ONLINE, WALK_UNBIASED)
from skywalker_b200.api import Context, DeviceArray, OfflineWalk, Sampler, Walker

APPS = {"deepwalk": APP_DEEPWALK, "ppr": APP_PPR, "node2vec": APP_NODE2VEC}
WALK_FLAGS = {"": 0, "unbiased": WALK_UNBIASED}
KHOP_RULES = {"replacement": 0, "take_all": KHOP_TAKE_ALL, "distinct": KHOP_DISTINCT, "unbiased": KHOP_UNBIASED}


def rmat(vertices, raw_edges, symmetric=False, weights="uniform"):
    return dict(graph="rmat", vertices=int(vertices), raw_edges=int(raw_edges), symmetric=symmetric, weights=weights)


def powerlaw(vertices, raw_edges, dmin=12.0, weights="uniform"):
    return dict(graph="powerlaw", vertices=int(vertices), raw_edges=int(raw_edges), dmin=dmin, cap=33000, weights=weights)


# The undirected power-law graph of benchmark configuration 3 (mean degree 76, hubs capped at 33,000).
POWERLAW_C3 = powerlaw(3070000, 117000000)


def listed():
    return [
        # Tables of a small graph (benchmark configuration 1): a call of this size is launches and host work.
        dict(name="build_small", kind="build", **rmat(1 << 16, 16 << 16)),
        # Tables of a large graph: the offline construction in bulk, every degree class in use.
        dict(name="build_large", kind="build", **rmat(1 << 24, 28 << 24)),
        # The weights of a resident graph have changed: its tables, the walk records and one batch of walks
        # (benchmark configuration 2: R-MAT 22, 40,000 walkers of 80 steps).
        dict(name="rebuild_and_walk", kind="rebuild", app="deepwalk", units=40000, length=80, **rmat(1 << 22, 16 << 22)),
        # The reference-shaped call on host arrays, a small batch: OfflineWalk over the table alone (sizes of
        # configuration 1, undirected so that every walk runs to its end).
        dict(name="offline_walk_host_small", kind="walk_rows", app="deepwalk", units=4096, length=80,
             **rmat(1 << 16, 16 << 16, symmetric=True)),
        # DeepWalk corpus for an embedding, device buffers, walk records; a ragged million walkers.
        dict(name="deepwalk_records", kind="walk", mode="offline", layout="records", app="deepwalk", units=999983, length=80,
             flags="", queued=False, **rmat(1 << 22, 16 << 22)),
        # Personalised PageRank by walks (configuration 5 with the graph two scales smaller): 8 M walkers, queued.
        dict(name="ppr_records_large", kind="walk", mode="offline", layout="records", app="ppr", units=8000000, length=100,
             flags="", queued=True, **rmat(1 << 24, 28 << 24)),
        # node2vec from prebuilt tables on the power-law graph.
        dict(name="node2vec_offline", kind="walk", mode="offline", layout="slots", app="node2vec", units=40000, length=80,
             flags="", queued=False, **POWERLAW_C3),
        # The same walks with no table at hand (configuration 3).
        dict(name="node2vec_online", kind="walk", mode="online", layout="slots", app="node2vec", units=40000, length=80,
             flags="", queued=False, **POWERLAW_C3),
        # Online 2-hop sampling, a full batch with replacement (configuration 4).
        dict(name="khop_online", kind="khop", mode="online", rule="replacement", units=65536, fanout="25,10",
             **rmat(4850000, 72000000)),
        # A mini-batch for a graph network: three hops from prebuilt tables, the offline sampler's take-all rule.
        dict(name="khop_offline_small", kind="khop", mode="offline", rule="take_all", units=1000, fanout="15,10,5",
             **rmat(4850000, 72000000)),
        # The online sampler's distinct-neighbour rule, host seeds in, packed tree out; an odd batch.
        dict(name="khop_distinct_host", kind="khop_packed", mode="online", rule="distinct", units=8191, fanout="25,10",
             **rmat(4850000, 72000000)),
        # PPR batch served to the host: starts in, byte lengths and packed walks out through pinned memory.
        dict(name="ppr_packed_host", kind="walk_packed", app="ppr", units=2000003, length=100, **rmat(1 << 22, 28 << 22)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _graph(rng, most_vertices, most_edges, symmetric=False):
    """Any vertex count, 4 to 28 raw edges a vertex (a power-law graph has up to 38, each stored both ways)."""
    weights = rng.choice(("uniform", "uniform", "lognormal"))
    if symmetric or rng.random() < 0.7:
        v = _log(rng, 1 << 14, most_vertices)
        return rmat(v, min(most_edges, v * rng.randint(4, 28)), symmetric, weights)
    v = _log(rng, 1 << 14, min(most_vertices, 3070000))
    return powerlaw(v, min(most_edges // 2, v * rng.randint(4, 38)), weights=weights)


def draw(rng):
    kind = rng.choice(("build", "build", "rebuild", "walk_rows", "walk", "walk", "walk", "online", "khop", "khop",
                       "khop_packed", "walk_packed"))
    length = rng.choice((rng.randint(5, 40), 80, rng.randint(41, 100)))
    if kind == "build":
        return dict(kind=kind, **_graph(rng, 1 << 24, 28 << 24))
    if kind == "rebuild":
        return dict(kind=kind, app=rng.choice(("deepwalk", "ppr")), units=_log(rng, 1000, 200000), length=length,
                    **_graph(rng, 1 << 22, 28 << 22))
    if kind == "walk_rows":
        return dict(kind=kind, app="deepwalk", units=_log(rng, 256, 40000), length=length,
                    **_graph(rng, 1 << 20, 16 << 20, symmetric=True))
    if kind == "walk":
        app = rng.choice(("deepwalk", "ppr", "node2vec"))
        units = _log(rng, 1000, {"deepwalk": 2000000, "ppr": 8000000, "node2vec": 100000}[app])
        layout = "slots" if app == "node2vec" else rng.choice(("records", "records", "slots"))
        return dict(kind=kind, mode="offline", layout=layout, app=app, units=units, length=length,
                    flags=rng.choice(("", "", "", "unbiased")), queued=rng.random() < 0.3, **_graph(rng, 1 << 23, 117000000))
    if kind == "online":
        return dict(kind="walk", mode="online", layout="slots", app=rng.choice(("deepwalk", "ppr", "node2vec")),
                    units=_log(rng, 256, 40000), length=min(length, 80), flags="", queued=False,
                    **_graph(rng, 4850000, 117000000))
    if kind in ("khop", "khop_packed"):
        fanout = rng.choice(("25,10", "25,10", "15,10,5", "10,5", "5,5,3", "40"))
        return dict(kind=kind, mode=rng.choice(("online", "offline")),
                    rule=rng.choice(("replacement", "take_all", "distinct", "unbiased")),
                    units=_log(rng, 100, 65536 if fanout in ("25,10", "10,5", "40") else 16384), fanout=fanout,
                    **_graph(rng, 4850000, 72000000))
    return dict(kind="walk_packed", app=rng.choice(("ppr", "ppr", "deepwalk")), units=_log(rng, 1000, 2000000),
                length=min(length, 20) if rng.random() < 0.5 else length, **_graph(rng, 1 << 22, 28 << 22))


# ---------------------------------------------------------------------------------------------------- prepare

def _resident_graph(case, seed):
    """A context with the case's graph resident; weights other than the generator's are a borrowed device array."""
    ctx = Context(0)
    s = seed * 7919 + 1
    if case["graph"] == "rmat":
        v = case["vertices"]
        scale = max(1, (v - 1).bit_length())
        ctx.generate_rmat(scale, case["raw_edges"], symmetric=case["symmetric"], graph_seed=1, weight_seed=s,
                          num_vertices=0 if v == 1 << scale else v)
    else:
        ctx.generate_powerlaw(case["vertices"], case["raw_edges"], 2.1, case["dmin"], case["cap"], 1, s)
    keep = []
    if case["weights"] != "uniform":
        V, E, _ = ctx.graph_info()
        x, a, _ = ctx.graph_device_ptrs()
        keep = [torch.as_tensor(DeviceArray(p, n, "<i4"), device="cuda").clone() for p, n in ((x, V + 1), (a, E))]
        g = torch.Generator(device="cuda").manual_seed(s)
        keep.append(torch.empty(E, device="cuda").log_normal_(0.0, 1.5, generator=g))
        torch.cuda.synchronize()
        ctx.adopt_device(V, E, *keep)
    return ctx, keep


def _start_vertices(ctx, n, seed, live):
    """Uniformly random start vertices; live: among those with out-edges."""
    V, E, _ = ctx.graph_info()
    g = torch.Generator(device="cuda").manual_seed(seed)
    if not live:
        return torch.randint(0, V, (n,), device="cuda", generator=g, dtype=torch.int32)
    x = torch.as_tensor(DeviceArray(ctx.graph_device_ptrs()[0], V + 1, "<i4"), device="cuda")
    have = torch.nonzero(x[1:] != x[:-1]).flatten().to(torch.int32)
    return have[torch.randint(0, len(have), (n,), device="cuda", generator=g)]


def _fanout(case):
    return [int(f) for f in case["fanout"].split(",")]


def prepare(case, seed):
    ctx, keep = _resident_graph(case, seed)
    kind = case["kind"]
    st = {"case": case, "ctx": ctx, "keep": keep, "seed": seed}
    online = case.get("mode") == "online" or case.get("flags") == "unbiased" or case.get("rule") == "unbiased"
    if kind not in ("build", "rebuild") and not online:
        ctx.alias_build_offline()  # the plan that such a program keeps
    if case.get("layout") == "records" or kind == "walk_packed":
        if online:
            ctx.alias_build_offline()
        ctx.walk_records_build()
    if kind == "build":
        torch.cuda.synchronize()
        return st
    n = case["units"]
    starts = _start_vertices(ctx, n, seed, live=kind == "walk_rows")
    if kind in ("walk", "rebuild"):
        st["starts"] = starts
        st["paths"] = torch.full((n, case["length"] + 1), -1, device="cuda", dtype=torch.int32)
        st["lengths"] = torch.zeros(n, device="cuda", dtype=torch.int32)
    elif kind == "walk_rows":
        st["walker"] = Walker(Sampler(None, ctx=ctx))
        st["walker"].seed = seed
        st["walker"].SetSeed(starts.cpu().numpy().view(np.uint32), case["length"] + 1)
    elif kind == "khop":
        cells, lens = ctx.khop_layout(_fanout(case))
        st["seeds"] = starts
        st["data"] = torch.full((n, cells), -1, device="cuda", dtype=torch.int32)
        st["lens"] = torch.zeros((n, lens), device="cuda", dtype=torch.int32)
    elif kind == "khop_packed":
        cells, lens = ctx.khop_layout(_fanout(case))
        st["seeds"] = starts.cpu().numpy().view(np.uint32)
        st["packed"] = torch.zeros(n * cells, dtype=torch.int32).pin_memory()
        st["lens"] = torch.zeros((n, lens), dtype=torch.int32).pin_memory()
    elif kind == "walk_packed":
        tp = 0.15 if case["app"] == "ppr" else 0.0
        most = n * (case["length"] + 1)
        st["starts"] = starts.cpu().pin_memory()
        st["packed"] = torch.zeros(min(most, int(n * (1 / tp + 2)) + 4096) if tp else most, dtype=torch.int32).pin_memory()
        st["lengths"] = torch.zeros(n, dtype=torch.uint8).pin_memory()
    torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------------------------------------------- run

def _walk(st):
    case, ctx = st["case"], st["ctx"]
    return ctx.walk(st["starts"], case["length"] + 1, app=APPS[case["app"]],
                    mode=MODE_ONLINE if case.get("mode") == "online" else MODE_OFFLINE,
                    tp=0.15, p=2.0, q=0.5, seed=st["seed"], paths=st["paths"], lengths=st["lengths"],
                    flags=WALK_FLAGS[case.get("flags", "")], enqueue_only=case.get("queued", False))


def _table(st):
    if "table" not in st:  # a view of the table that the context owns
        slots, valid = st["ctx"].alias_device_arrays()
        st["table"] = {"slots": torch.as_tensor(slots, device="cuda"), "valid": torch.as_tensor(valid, device="cuda")}
    return st["table"]


def run(st):
    case, ctx, kind = st["case"], st["ctx"], st["case"]["kind"]
    if kind == "build":
        ctx.alias_build_offline()
        return _table(st)
    if kind == "rebuild":
        ctx.alias_build_offline()
        ctx.walk_records_build()
        paths, lengths, _, edges = _walk(st)
        return dict(_table(st), paths=paths, lengths=lengths, edges=edges)
    if kind == "walk":
        paths, lengths, _, edges = _walk(st)
        return {"paths": paths, "lengths": lengths, "edges": edges}
    if kind == "walk_rows":
        OfflineWalk(st["walker"])
        return {"paths": st["walker"].result.data, "lengths": st["walker"].result.length, "edges": st["walker"].sampled_edges}
    if kind == "khop":
        data, lens, _, edges = ctx.sample_khop(st["seeds"], _fanout(case),
                                               mode=MODE_ONLINE if case["mode"] == "online" else MODE_OFFLINE,
                                               flags=KHOP_RULES[case["rule"]], seed=st["seed"], data=st["data"],
                                               sample_lengths=st["lens"])
        return {"data": data, "lens": lens, "edges": edges}
    if kind == "khop_packed":
        packed, lens, cells, _, edges = ctx.sample_khop_packed(
            st["seeds"], _fanout(case), mode=MODE_ONLINE if case["mode"] == "online" else MODE_OFFLINE,
            flags=KHOP_RULES[case["rule"]], seed=st["seed"], packed=st["packed"], sample_lengths=st["lens"])
        return {"packed": packed, "cells": cells, "lens": lens, "edges": edges}
    packed, lengths, cells, _, edges = ctx.walk_packed(st["starts"], case["length"] + 1, app=APPS[case["app"]], tp=0.15,
                                                       seed=st["seed"], packed=st["packed"], lengths=st["lengths"],
                                                       n=case["units"], lengths_u8=True)
    return {"packed": packed, "cells": cells, "lengths": lengths, "edges": edges}


# ------------------------------------------------------------------------------------------- work and tolerance

def _edges(case):
    """About how many edges are stored: nearly every raw edge survives the removal of loops and duplicates."""
    return int(case["raw_edges"] * 0.95) * (2 if case["graph"] == "powerlaw" or case["symmetric"] else 1)


def _steps(case):
    """About how many steps a walk makes.  Uniformly random starts on a directed R-MAT graph are mostly dead ends
    (a DeepWalk makes 0.38 of its steps, a PPR walk at tp = 0.15 makes 2.6); elsewhere walks rarely end early."""
    directed = case["graph"] == "rmat" and not case["symmetric"]
    if case["app"] == "ppr":
        return min(case["length"], 2.6 if directed else (1 - 0.15) / 0.15)
    return case["length"] * (0.38 if directed else 1.0)


def work(case):
    """Bytes of one pass, each input read once and each output written once: 12 an edge of a table (weight in, slot
    out), 24 a step (offset pair, slot, neighbour, path cell), 8 a walker (start, length; a byte length for packed
    results), 8 a tree cell that holds a sample (neighbour, cell), 4 a length.  An online draw reads a weight in the
    slot's place.  Operations: the quantise-scan-merge chain of a table edge, the counter-based generator of a draw."""
    kind, b, f = case["kind"], 0.0, 0.0
    if kind in ("build", "rebuild"):
        b += 12.0 * _edges(case) + 5.0 * case["vertices"]
        f += 40.0 * _edges(case)
    if kind in ("rebuild", "walk", "walk_rows", "walk_packed"):
        steps = case["units"] * _steps(case)
        b += 24.0 * steps + (5.0 if kind == "walk_packed" else 8.0) * case["units"]
        f += 80.0 * steps
    if kind in ("khop", "khop_packed"):
        width, parents = 1, 0.0
        filled = 1.0 if case["graph"] == "powerlaw" else 0.55  # a directed R-MAT graph has dead ends
        for fan in _fanout(case):
            parents += width
            width = width * fan * filled
            b += case["units"] * width * 24.0
            f += case["units"] * width * 80.0
        b += 4.0 * case["units"] * (1 + parents)
    return {"bytes": b, "flops": f}


def tolerance(case):
    return "exact"
