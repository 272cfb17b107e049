"""Timed cases of the temporal-motif miner: what a program that uses it has it do.

A case names a graph shape and the queries one pass runs on it.  The graphs
follow the two families of ``everest_b200/synth.py`` (the same laws, drawn on
the GPU so that inputs are quick to make): ``zipf`` has uniform timestamps,
``bursty`` has power-law senders that write in bursts and are answered.

kind         one pass
``count``    every pattern of the set, one at a time, on a resident graph
``batch``    the same queries handed over as one batch
``rows``     an enumeration, its rows read back and put in order
``cons``     queries under node predicates, time gaps, anti-edges and a filter
``load``     host arrays to a resident graph, a few counts, graph freed
"""
import math

import numpy as np
import torch

from everest_b200 import capi, synth, workloads
from everest_b200.constraints import Constraints

DEV = 0
T_ZIPF = 10_000_000       # zipf family: timestamps uniform in [0, T_ZIPF)
T_BURSTY = 230_000_000    # bursty family: burst starts uniform in [0, T_BURSTY)
GAP_US = 60e6             # mean gap inside a burst
REPLY = 0.25              # share of a burst's edges that answer its source


def listed():
    return [
        # one small question to a small graph: launch and latency count
        dict(name="triangle-200k", kind="count", family="zipf", nodes=10_000, edges=200_000, patterns="triangle",
             delta=3600, window=0, strict=False),
        # one request of a service: a four-edge motif over a short stretch of time
        dict(name="window-1k", kind="count", family="bursty", nodes=140_000, edges=1_000_003, patterns="4-cycle",
             delta=86400, window=1000, strict=False),
        # the motif census of a message graph, every three-edge pattern on its own
        dict(name="census-3edge-7.8m", kind="count", family="bursty", nodes=1_100_000, edges=7_800_000,
             patterns="three-edge", delta=86400, window=0, strict=False),
        # larger patterns over the same graph
        dict(name="patterns-4edge-7.8m", kind="count", family="bursty", nodes=1_100_000, edges=7_800_000,
             patterns="random-8-4-4-11", delta=86400, window=0, strict=False),
        # five-edge patterns, an odd number of edges, strictly rising times
        dict(name="patterns-5edge-1.3m", kind="count", family="bursty", nodes=183_001, edges=1_299_827,
             patterns="random-6-5-5-12", delta=14400, window=0, strict=True),
        # the largest single question: round trips in a large graph
        dict(name="4-cycle-36m", kind="count", family="bursty", nodes=2_600_000, edges=36_000_000,
             patterns="4-cycle", delta=86400, window=0, strict=False),
        # an analyst's batch: mixed sizes and windows of time in one call
        dict(name="batch-64-7.8m", kind="batch", family="bursty", nodes=1_100_000, edges=7_800_000,
             patterns="random-64-3-4-3", delta=0, window=250_000, strict=False, tile=256, graph=True),
        # what a serving loop hands over at once: many short requests
        dict(name="serve-64-7.8m", kind="batch", family="bursty", nodes=1_100_000, edges=7_800_000,
             patterns="random-64-3-5-5", delta=-1, window=1000, strict=False, tile=64, graph=False),
        # all matches of a small graph, read back
        dict(name="rows-triangle-200k", kind="rows", family="zipf", nodes=10_000, edges=200_000, patterns="triangle",
             delta=3600, window=0, strict=False, cap=1_000_000),
        # all round trips that start in a stretch of a larger graph
        dict(name="rows-4-cycle-7.8m", kind="rows", family="bursty", nodes=1_100_000, edges=7_800_000,
             patterns="4-cycle", delta=86400, window=500_000, strict=False, cap=1_000_000),
        # conditions on nodes, times, missing edges and whole matches
        dict(name="constrained-7.8m", kind="cons", family="bursty", nodes=1_100_000, edges=7_800_000,
             patterns="constrained", delta=86400, window=0, strict=False),
        # a graph comes in from the host and is asked at once
        dict(name="load-7.8m", kind="load", family="bursty", nodes=1_100_000, edges=7_800_000, patterns="triangle",
             delta=86400, window=0, strict=False),
    ]


def draw(rng):
    """A case of the same ranges: sizes over their logarithm, odd ones too."""
    kind = rng.choice(["count", "count", "batch", "batch", "rows", "cons", "load"])
    family = "zipf" if kind in ("count", "rows", "load") and rng.random() < 0.3 else "bursty"
    top = 400_000 if family == "zipf" else 7_800_000
    edges = int(math.exp(rng.uniform(math.log(20_000), math.log(top))))
    c = dict(kind=kind, family=family, nodes=max(500, edges // rng.choice([7, 11, 20])), edges=edges, window=0,
             strict=rng.random() < 0.25)
    day = int(math.exp(rng.uniform(math.log(600), math.log(86400 if family == "bursty" else 3600))))
    seed = rng.randrange(1 << 20)
    if kind == "count":
        k = rng.choice([2, 3, 3, 4, 4] if family == "zipf" else [2, 3, 3, 4, 4, 5])
        c.update(patterns="random-%d-%d-%d-%d" % (1 if k == 2 else rng.choice([1, 4]), k, k, seed),
                 delta=min(day, 3600) if k == 5 else day)
        if rng.random() < 0.4:
            c.update(window=int(math.exp(rng.uniform(math.log(500), math.log(edges)))))
    elif kind == "batch":
        c.update(patterns="random-%d-3-4-%d" % (rng.choice([5, 16, 33, 64]), seed), delta=day, graph=rng.random() < 0.5,
                 tile=rng.choice([64, 128, 256]), window=int(math.exp(rng.uniform(math.log(500), math.log(200_000)))))
    elif kind == "rows":
        c.update(patterns=rng.choice(["triangle", "triangle" if family == "zipf" else "4-cycle"]), cap=1_000_000,
                 delta=min(day, 14400), window=rng.randrange(1000, 100_000))
    elif kind == "cons":
        c.update(patterns="constrained", delta=day, strict=False)
    else:
        c.update(patterns="triangle", delta=day)
    return c


# ------------------------------------------------------------------ inputs --

def _power_law(n, s):
    w = np.cumsum(np.arange(1, n + 1, dtype=np.float64) ** -s)
    return torch.from_numpy(w / w[-1]).cuda()


def _edges(case, seed):
    """u, v, t sorted by time (int64, on the GPU), vertices numbered by first
    appearance, and their number: what the loader makes of an edge list."""
    g = torch.Generator("cuda").manual_seed(seed)
    n, e = case["nodes"], case["edges"]

    def rand(k):
        return torch.rand(k, generator=g, device="cuda", dtype=torch.float64)

    zipf = case["family"] == "zipf"
    cdf = _power_law(n, 1.5 if zipf else 1 / 1.1)

    def node(k):
        return torch.searchsorted(cdf, rand(k), right=True).clamp_(max=n - 1)

    if zipf:
        u, v = node(e), node(e)
        t = (rand(e) * T_ZIPF).long()
    else:
        sizes = torch.poisson(torch.full((e // 20 + e // 100 + 64,), 20.0, device="cuda"), generator=g).long().clamp_(min=1)
        burst = torch.repeat_interleave(torch.arange(sizes.numel(), device="cuda"), sizes)[:e]
        e = burst.numel()
        first = (sizes.cumsum(0) - sizes)[burst]
        u, v = node(sizes.numel())[burst], node(e)
        gaps = (-torch.log1p(-rand(e)) * GAP_US).long().cumsum(0)
        t = (rand(sizes.numel()) * T_BURSTY * 1e6).long()[burst] + gaps - gaps[first]
        t //= 1_000_000
    bad = u == v
    v = torch.where(bad, (v + 1 + (rand(v.numel()) * (n - 1)).long()) % n, v)
    if not zipf:
        i = torch.arange(e, device="cuda")
        reply = (rand(e) < REPLY) & (i > first)
        asked = torch.where(reply, -1, i).cummax(0).values
        u, v = torch.where(reply, v[asked], u), torch.where(reply, u, v)
    t, order = t.sort(stable=True)
    u, v = u[order], v[order]
    seen = torch.full((n,), 1 << 62, device="cuda", dtype=torch.int64)
    seen.scatter_reduce_(0, torch.stack([u, v], 1).reshape(-1), torch.arange(2 * e, device="cuda"), "amin")
    rank = torch.empty_like(seen)
    rank[seen.argsort()] = torch.arange(n, device="cuda")
    return rank[u], rank[v], t, int((seen < 1 << 62).sum())


def _arrays(case, seed):
    """The graph arrays of the C ABI, on the GPU."""
    u, v, t, n = _edges(case, seed)

    def lists(x):
        order = x.sort(stable=True).indices.int()
        offsets = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        offsets[1:] = torch.bincount(x, minlength=n).cumsum(0)
        return order, offsets.int()

    (out_v, out_r), (in_v, in_r) = lists(u), lists(v)
    eg = torch.stack([u, v, t], 1).int().reshape(-1)
    euid = torch.arange(u.numel(), device="cuda", dtype=torch.int32)
    return u.numel(), n, eg, out_v, in_v, out_r, in_r, euid


def _patterns(case):
    p = case["patterns"]
    if p == "triangle":
        return [([0, 1, 2], [1, 2, 0])]
    if p == "4-cycle":
        return [([0, 1, 2, 3], [1, 2, 3, 0])]
    if p == "three-edge":
        sets = synth.three_edge_patterns()
    else:
        count, lo, hi, seed = (int(x) for x in p.split("-")[1:])
        sets = synth.random_patterns(count, (lo, hi), (2, 4 if hi > 2 else 3), seed)
    return [([a for a, _ in s], [b for _, b in s]) for s in sets]


def _queries(case, seed, edges):
    """(mu, mv, delta, beg, end) of one pass.  delta 0 goes through hours,
    days and weeks, -1 is spread over minutes to a day."""
    r = np.random.default_rng([seed, 7])
    fixed = np.random.default_rng(case["edges"])  # a case's windows of time do not change with the seed
    out = []
    for i, (mu, mv) in enumerate(_patterns(case)):
        d = case["delta"]
        if d == 0:
            d = (3600, 86400, 604800)[i % 3]
        elif d < 0:
            d = int(math.exp(fixed.uniform(math.log(600), math.log(86400))))
        if case["window"]:
            beg = int(r.integers(0, max(1, edges - case["window"])))
            out.append((mu, mv, d, beg, min(edges, beg + case["window"])))
        else:
            out.append((mu, mv, d, 0, -1))
    return out


def _constrained(case):
    """The feature queries of the benchmark, gaps in proportion to delta."""
    out = []
    for _, mu, mv, cons in workloads.constrained_queries():
        cons = dict(cons)
        if "temporal" in cons:
            cons["temporal"] = [x * case["delta"] // cons["delta"] for x in cons["temporal"]]
        out.append((mu, mv, Constraints.from_yaml(cons, mu, mv)))
    return out


def prepare(case, seed):
    edges, nodes, *arrays = _arrays(case, seed)
    s = {"case": case, "flags": capi.FLAG_STRICT_TS if case["strict"] else 0}
    if case["kind"] == "load":
        s["host"] = capi.HostGraph(edges, nodes, *(x.cpu().pin_memory().numpy() for x in arrays))
    else:
        torch.cuda.synchronize()
        s["graph"] = capi.DeviceGraph.from_device(DEV, edges, nodes, *(x.data_ptr() for x in arrays))
    if case["kind"] == "batch":
        s["batch"] = capi.Batch(DEV, 64)
        s["batch"].set_tuning(tile_roots=case["tile"], use_graph=case["graph"])
    else:
        s["worker"] = capi.Worker(DEV)
    if case["kind"] == "cons":
        r = np.random.default_rng([seed, 8])
        s["graph"].set_features(r.integers(0, 10**9, nodes), r.integers(0, 10**9, edges))
        s["queries"] = _constrained(case)
    else:
        s["queries"] = _queries(case, seed, edges)
    return s


# --------------------------------------------------------------- one pass --

def run(s):
    kind = s["case"]["kind"]
    if kind == "batch":
        b = s["batch"]
        b.clear()
        for mu, mv, delta, beg, end in s["queries"]:
            b.add(s["graph"], mu, mv, delta, beg, end, s["flags"])
        return np.array(b.run(), np.int64)
    w = s["worker"]
    if kind == "cons":
        out = []
        for mu, mv, cons in s["queries"]:
            w.take(s["graph"], mu, mv, s["case"]["delta"], constraints=cons)
            out.append(w.run())
        return np.array(out, np.int64)
    if kind == "rows":
        (mu, mv, delta, beg, end), = s["queries"]
        w.take(s["graph"], mu, mv, delta, beg, end, s["case"]["cap"], s["flags"])
        n = w.run()
        return {"count": n, "rows": _in_order(w.enum_rows(n), s["case"]["cap"])}
    graph = s["graph"] if kind == "count" else capi.DeviceGraph(s["host"], DEV)
    out = []
    for mu, mv, delta, beg, end in s["queries"]:
        w.take(graph, mu, mv, delta, beg, end, 0, s["flags"])
        out.append(w.run())
    if kind == "load":
        graph.free()
    return np.array(out, np.int64)


def _in_order(rows, cap):
    """Matches come in no fixed order; a program that compares or stores them
    sorts them (by their edges, first to last), here into a table of cap rows."""
    r = torch.from_numpy(rows).cuda().long()
    low = r[:, -1] if r.shape[1] == 3 else r[:, 2] << 32 | r[:, 3]
    order = low.argsort()
    table = torch.full((cap, r.shape[1]), -1, device="cuda")
    table[: len(r)] = r[order[(r[order, 0] << 32 | r[order, 1]).argsort(stable=True)]]
    return table


def work(case):
    """Each question reads the edges of its stretch of time (u, v, t) once and
    writes a count (its rows); a graph that comes in is read once."""
    e = min(case["edges"], case["window"] or case["edges"])
    if case["kind"] == "cons":
        n, extra = len(workloads.constrained_queries()), 4 * (case["nodes"] + e)
    else:
        n, extra = len(_patterns(case)), 0
    if case["kind"] == "load":
        extra = 24 * e + 8 * (case["nodes"] + 1)
    return {"bytes": n * (12 * e + 8 + extra), "flops": 0}


# ---------------------------------------------------------------- 64 bits --

def _matches(edges, mu, mv, delta, beg, end, strict):
    """Every match, as rows of edge numbers: the partial matches of one edge
    joined with all later edges at a mapped node inside the window."""
    u, v, t = edges
    e = u.numel()
    keys = [(x * e + torch.arange(e, device=x.device)).sort().values for x in (u, v)]
    rows = []
    for b in range(beg, end, 20_000):
        ids = torch.arange(b, min(end, b + 20_000), device=u.device)
        ids = ids[u[ids] != v[ids]]
        nodes, found = {0: u[ids], 1: v[ids]}, [ids]
        stop = torch.searchsorted(t, t[ids] + delta, right=True)
        for a, c in zip(mu[1:], mv[1:]):
            at = found[-1] + 1
            if strict:
                at = torch.searchsorted(t, t[found[-1]], right=True)
            base, key = (nodes[a], keys[0]) if a in nodes else (nodes[c], keys[1])
            lo, hi = torch.searchsorted(key, base * e + at), torch.searchsorted(key, base * e + stop)
            n = (hi - lo).clamp_(min=0)
            one = torch.repeat_interleave(torch.arange(n.numel(), device=u.device), n)
            new = key[(lo - (n.cumsum(0) - n))[one] + torch.arange(one.numel(), device=u.device)] % e
            ends = {a: u[new], c: v[new]}
            ok = torch.ones_like(new, dtype=torch.bool)
            for m, x in ends.items():
                for q, y in nodes.items():
                    ok &= (y[one] == x) if q == m else (y[one] != x)
            one, new = one[ok], new[ok]
            nodes = {q: y[one] for q, y in nodes.items()} | {m: x[ok] for m, x in ends.items()}
            found, stop = [f[one] for f in found] + [new], stop[one]
        rows.append(torch.stack(found, 1))
    return torch.cat(rows)


def exact(case, seed):
    """By joins, where the graph is small and the patterns are short."""
    if case["kind"] == "cons" or case["edges"] > 400_000 or case["patterns"] not in ("triangle", "4-cycle"):
        return None
    *edges, _ = _edges(case, seed)
    e = edges[0].numel()
    out = []
    for mu, mv, delta, beg, end in _queries(case, seed, e):
        out.append(_matches(edges, mu, mv, delta, beg, e - len(mu) + 1 if end < 0 else end, case["strict"]))
    if case["kind"] == "rows":
        return {"count": len(out[0]), "rows": _in_order(out[0].cpu().numpy(), case["cap"])}
    return np.array([len(x) for x in out], np.int64)
