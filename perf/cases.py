"""The work this framework is asked to do, as cases that can be timed.

A case names one public entry point, a data graph and the queries asked of it.
The data graph is part of the case (it stays resident, as the handle a user's
program keeps) and the queries come from the seed: random walks over that
graph, as everywhere in this repository. Whole-number results (rows, counts,
orders, CSR arrays) are compared value by value; only the join-order model's
gradient is a computed number.

Graph and query shapes are those of gpsm_b200/workloads.py (small_er, rmat20,
rmat20_mix, rmat22) and of the tests; the caps are the benchmark's or smaller,
with a work cap where a single unlucky query could otherwise run for minutes
(and low enough that some queries of a batch stop there: a batch returns counts
and how each query ended).
"""
import math
import random
from collections import OrderedDict

import numpy as np
import torch

import gpsm_b200 as G
from gpsm_b200 import learned
from gpsm_b200 import workloads as W

MODES = {"induced": W.MODE_INDUCED, "tree": W.MODE_TREE, "dense": W.MODE_DENSE}

ER = dict(graph="er", n=10_000, m=40_000, labels=8, zipf=0.0)
RMAT20 = dict(graph="rmat", n=1 << 20, m=16 << 20, labels=32, zipf=1.0)
RMAT22 = dict(graph="rmat", n=1 << 22, m=64 << 20, labels=64, zipf=1.1)


def listed():
    return [
        # one small query on a small graph, every row returned: the reference's own run.cpp call, all latency
        dict(name="match_er_6", kind="match", **ER, queries=1, qlo=6, qhi=6, mode="induced", min_deg=0.0, cap=0,
             work_cap=0, order="plain", directed=False),
        # a stream of small queries one after another on one engine: launches and host round trips
        dict(name="batch_er_64", kind="batch", **ER, queries=64, qlo=4, qhi=8, mode="mix", min_deg=0.0, cap=0,
             work_cap=0, order="plain", slots=1),
        # directed, edge-labelled queries (the reference's verify) on a middle-sized graph, rows returned
        dict(name="match_directed_rmat16", kind="match", graph="rmat", n=1 << 16, m=1 << 20, labels=16, zipf=1.0,
             queries=3, qlo=3, qhi=5, mode="tree", min_deg=0.0, cap=100_000, work_cap=0, order="plain",
             directed=True),
        # the rmat20 benchmark query with its rows on the host
        dict(name="match_rmat20_12", kind="match", **RMAT20, queries=1, qlo=12, qhi=12, mode="induced", min_deg=2.5,
             cap=1_000_000, work_cap=1 << 30, order="plain", directed=False),
        # candidate sets, candidate edges and the plain order alone: what order training and admission ask for
        dict(name="filter_rmat22_24", kind="filter", **RMAT22, queries=2, qlo=23, qhi=24, mode="dense", min_deg=0.0),
        # the rmat20 benchmark batch in the reference's order on one engine
        dict(name="batch_rmat20_12", kind="batch", **RMAT20, queries=12, qlo=12, qhi=12, mode="induced", min_deg=2.5,
             cap=10_000_000, work_cap=80_000_000, order="plain", slots=1),
        # the mixed 4..32-vertex set in the learned order on all engine slots
        dict(name="batch_rmat20_mix", kind="batch", **RMAT20, queries=32, qlo=4, qhi=32, mode="mix", min_deg=0.0,
             cap=10_000_000, work_cap=1 << 27, order="learned", slots=12),
        # the headline batch: large queries on the large graph, learned order, all engine slots
        dict(name="batch_rmat22_mix", kind="batch", **RMAT22, queries=24, qlo=4, qhi=64, mode="mix", min_deg=0.0,
             cap=10_000_000, work_cap=1 << 28, order="learned", slots=12),
        # one large dense query on the large graph, counted alone on an idle GPU
        dict(name="count_rmat22_40", kind="count", **RMAT22, queries=2, qlo=36, qhi=40, mode="mix", min_deg=0.0,
             cap=10_000_000, work_cap=1 << 30, order="learned"),
        # the request server: rows of every request back in host memory, collected as they finish
        dict(name="serve_rmat20_mix", kind="serve", **RMAT20, queries=16, qlo=4, qhi=24, mode="mix", min_deg=0.0,
             cap=200_000, work_cap=1 << 28, order="learned", slots=4),
        # a data graph built from its edge list and read back
        dict(name="build_rmat18", kind="build", graph="rmat", n=1 << 18, m=4 << 20, labels=32, zipf=1.0),
        # the join-order model's loss and gradient over a training set's share
        dict(name="grad_16384", kind="grad", samples=16384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["match", "match", "batch", "batch", "batch", "filter", "count", "serve", "build", "grad"])
    if kind == "grad":
        return dict(kind="grad", samples=_log(rng, 300, 40_000))
    if kind == "build":
        n = _log(rng, 1000, 300_000)
        return dict(kind="build", graph=rng.choice(["er", "rmat"]), n=n, m=n * rng.randint(2, 14),
                    labels=_log(rng, 4, 64), zipf=rng.choice([0.0, 1.0]))
    which = rng.choice(["er", "rmat", "rmat", "rmat20", "rmat22"])
    if kind == "serve" and which == "rmat22":
        which = "rmat"
    if which == "er":
        n = _log(rng, 2_000, 60_000)
        c = dict(graph="er", n=n, m=int(n * rng.uniform(2.5, 5.0)), labels=rng.randint(6, 16), zipf=0.0)
    elif which == "rmat":
        n = _log(rng, 1 << 14, 600_000)
        c = dict(graph="rmat", n=n, m=n * rng.randint(6, 16), labels=rng.randint(16, 48),
                 zipf=rng.choice([0.5, 1.0]))
    else:
        c = dict(RMAT20 if which == "rmat20" else RMAT22)
    # the largest queries go with the largest graphs
    qtop = {"er": 9, "rmat": 20, "rmat20": 30, "rmat22": 60}[which]
    qlo = rng.randint(3, max(4, qtop // 2))
    qhi = min(qtop, qlo + rng.randint(0, qtop // 2))
    c = dict(kind=kind, **c, qlo=qlo, qhi=qhi, mode=rng.choice(["tree", "dense", "mix"]), min_deg=0.0)
    if kind == "filter":
        return dict(c, queries=rng.randint(1, 2))
    order = rng.choice(["plain", "learned"])
    if kind == "match":
        if which in ("er", "rmat") and c["n"] < 100_000 and rng.random() < 0.5:  # few rows pass: small trees
            return dict(c, qlo=rng.randint(3, 4), qhi=rng.randint(4, 5), mode="tree", queries=rng.randint(1, 3),
                        cap=_log(rng, 1_000, 100_000), work_cap=0, order=order, directed=True)
        return dict(c, queries=rng.randint(1, 3), cap=_log(rng, 1_000, 500_000), work_cap=1 << 28, order=order,
                    directed=False)
    if kind == "count":
        return dict(c, queries=rng.randint(1, 2), cap=_log(rng, 10_000, 10_000_000), work_cap=1 << 29, order=order)
    if kind == "batch":
        cap = rng.choice([0, 10_000_000])  # under the cap a lower work cap, so that not every count is the cap
        return dict(c, queries=rng.randint(6, 24), cap=cap, work_cap=_log(rng, 1 << 20, 1 << (23 if cap else 26)),
                    order=order, slots=rng.choice([1, 12]))
    return dict(c, queries=rng.randint(4, 16), cap=_log(rng, 1_000, 200_000), work_cap=1 << 28, order=order, slots=4)


# ---- data graphs: made once per process from the case, kept like any resident handle ----

_graphs = OrderedDict()  # (graph, n, m, labels, zipf, directed) -> (host graph, device graph)
_models = []


def _pair_bits(a, b):
    """(whether the undirected pair (a < b) points from b to a, its edge label 1..2), fixed by the pair alone."""
    x = a.astype(np.uint64) * np.uint64(2654435761) + b.astype(np.uint64) * np.uint64(40503)
    return ((x >> np.uint64(7)) & np.uint64(1)).astype(bool), (1 + ((x >> np.uint64(12)) & np.uint64(1))).astype(np.uint32)


def _edges(kind, n, m, seed):
    """About m unique undirected edges (u < v) over n vertices, uint32 [m, 2] on the host."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    bits = max(1, (n - 1).bit_length())
    relabel = torch.randperm(1 << bits, generator=g, device="cuda")
    keys = torch.zeros(0, dtype=torch.int64, device="cuda")
    for _ in range(12):
        k = int((m - keys.numel()) * 1.4) + 1024
        if kind == "rmat":  # quadrant probabilities .57 .19 .19 .05
            u = torch.zeros(k, dtype=torch.int64, device="cuda")
            v = torch.zeros(k, dtype=torch.int64, device="cuda")
            for _ in range(bits):
                r = torch.rand(k, generator=g, device="cuda")
                u.mul_(2).add_(r >= 0.76)
                v.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
            u, v = relabel[u] % n, relabel[v] % n
        else:
            u = torch.randint(n, (k,), generator=g, device="cuda")
            v = torch.randint(n, (k,), generator=g, device="cuda")
        lo, hi = torch.minimum(u, v), torch.maximum(u, v)
        keys = torch.unique(torch.cat([keys, (lo * (1 << 32) + hi)[lo < hi]]))
        if keys.numel() >= m:
            break
    if keys.numel() > m:
        keys = keys[torch.randperm(keys.numel(), generator=g, device="cuda")[:m]]
    e = torch.stack([keys >> 32, keys & 0xFFFFFFFF], 1).to(torch.int32).cpu().numpy().view(np.uint32)
    del relabel, keys
    torch.cuda.empty_cache()
    return e


def _labels(n, labels, zipf, seed):
    p = 1.0 / np.arange(1, labels + 1) ** zipf
    return np.random.default_rng(seed).choice(labels, size=n, p=p / p.sum()).astype(np.uint32) + 1


def _graph(c):
    key = (c["graph"], c["n"], c["m"], c["labels"], c["zipf"], bool(c.get("directed")))
    if key in _graphs:
        _graphs.move_to_end(key)
        return _graphs[key]
    while len(_graphs) >= 6:
        _graphs.popitem(last=False)
    salt = c["n"] * 31 + c["m"] * 7 + c["labels"]
    g = W.Graph(c["n"], None, None, _labels(c["n"], c["labels"], c["zipf"], salt),
                _edges(c["graph"], c["n"], c["m"], salt + 1), c["graph"])
    dg = G.DeviceGraph(g, build_on_device=True)
    g.offsets, g.cols = dg.download()
    if c.get("directed"):
        back, lab = _pair_bits(g.edges[:, 0], g.edges[:, 1])
        dg.set_directed(np.where(back[:, None], g.edges[:, ::-1], g.edges), lab)
    _graphs[key] = (g, dg)
    return _graphs[key]


def _model():
    if not _models:
        _models.append(learned.load(0))
    return _models[0]


def _queries(c, g, seed):
    """Random-walk queries of evenly spread sizes; those of "mix" are trees and dense ones in turn."""
    rng = random.Random(seed * 7919 + 13)
    out = []
    for k in range(c["queries"]):
        mode = c["mode"] if c["mode"] != "mix" else ("tree", "dense")[k % 2]
        n = c["qlo"] + round(k * (c["qhi"] - c["qlo"]) / max(1, c["queries"] - 1))
        for _ in range(400):
            try:
                q = W.random_walk_query(g, n, rng.getrandbits(60), MODES[mode], 0.3, c["min_deg"])
                break
            except G.GpsmError:  # the walk got stuck (or no such dense spot): another start
                pass
        else:
            raise RuntimeError("no query of %d vertices found" % n)
        elab = None
        if c.get("directed"):  # the walked data edges' own directions and labels
            a, b = q.data_ids[q.edges[:, 0]], q.data_ids[q.edges[:, 1]]
            back, elab = _pair_bits(np.minimum(a, b), np.maximum(a, b))
            turn = (a > b) != back
            q.edges = np.ascontiguousarray(np.where(turn[:, None], q.edges[:, ::-1], q.edges))
        out.append((q, elab))
    return out


class _Params:
    """Weights of the 16-64-64-1 model and its training samples, from a seed."""

    def __init__(self, c, seed):
        r = np.random.default_rng(seed)
        n, f, h = c["samples"], 16, 64
        self.w = np.concatenate([
            r.uniform(-1, 1, h * f) * math.sqrt(6 / f), r.normal(0, 0.1, h),
            r.uniform(-1, 1, h * h) * math.sqrt(6 / h), r.normal(0, 0.1, h),
            r.uniform(-1, 1, h) * math.sqrt(6 / h), r.normal(0, 0.1, 1)]).astype(np.float32)
        self.x = r.gamma(2.0, 2.0, (n, f)).astype(np.float32)  # log2 counts, degrees and sizes: positive, skewed
        self.y = r.normal(1.0, 3.0, n).astype(np.float32)  # log2 expansion of a join step


def prepare(case, seed):
    G.init(0)
    kind = case["kind"]
    s = {"case": case}
    if kind == "grad":
        s["p"] = _Params(case, seed)
        s["model"] = G.Model(0, params=s["p"].w)
        return s
    if kind == "build":
        s["graph"] = W.Graph(case["n"], None, None, _labels(case["n"], case["labels"], case["zipf"], seed + 5),
                             _edges(case["graph"], case["n"], case["m"], seed))
        return s
    g, s["dg"] = _graph(case)
    s["q"] = _queries(case, g, seed)
    s["model"] = _model() if case.get("order") == "learned" else None
    if kind in ("match", "serve"):  # where rows go that are fewer than the cap
        s["rows"] = [np.zeros((case["cap"] or 1 << 16, q.n), np.int32) for q, _ in s["q"]]
    if kind == "batch":
        s["list"] = [q for q, _ in s["q"]]
        s["packed"] = G.pack_queries(s["list"])
    if kind == "serve":
        s["server"] = G.Server(s["dg"], slots=case["slots"], slot_arena=4 << 30, cap=case["cap"],
                               order="learned" if s["model"] else None, model=s["model"], collect_rows=True,
                               work_cap=case["work_cap"])
    return s


def _ints(a):
    return np.ascontiguousarray(a).view(np.int32)  # the same 32 bits


def _table(rows, into):
    """The rows as the call returned them, or, when the query has fewer than the cap, at the start of `into`
    (zeros after them), so that a case's outputs always have one shape."""
    if len(rows) == len(into):
        return _ints(rows)
    k = min(len(rows), len(into))
    into[:k] = _ints(rows)[:k]
    return into


def _padded(a, n):
    out = np.zeros(n, np.int64)
    out[: len(a)] = a
    return out


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "grad":
        loss, g = state["model"].grad(state["p"].x, state["p"].y)
        return {"loss": loss, "grad": g}
    if kind == "build":
        dg = G.DeviceGraph(state["graph"], build_on_device=True)
        off, cols = dg.download()
        slots = dg.edge_table()[0]
        dg.free()
        return {"offsets": _ints(off), "cols": _ints(cols), "table_slots": slots}
    dg, model = state["dg"], state["model"]
    order = "learned" if model else None
    if kind == "filter":
        out = []
        for q, _ in state["q"]:
            f = G.debug_filter(dg, q)
            pairs = q.n * (q.n - 1) // 2  # dense queries differ in their number of edges
            out.append([_ints(f["cand_count"]), _padded(f["size_fwd"], pairs), _padded(f["size_rev"], pairs),
                        _ints(f["filter_order"]), f["plain_pos2id"], f["empty"]])
        return out
    if kind == "batch":
        counts, capped, _, info = G.match_batch(dg, state["list"], cap=c["cap"] or None, orders=order,
                                                packed=state["packed"], slots=c["slots"], model=model,
                                                slot_arena=13 << 29 if c["slots"] > 1 else 0, work_cap=c["work_cap"])
        return {"counts": counts.astype(np.int64), "stop": info["stop"]}
    if kind == "serve":
        srv = state["server"]
        tickets = [srv.submit(q)[0] for q, _ in state["q"]]
        at = {t: i for i, t in enumerate(tickets)}
        out = [None] * len(tickets)
        for _ in tickets:
            (t, _), r = srv.wait_any()
            out[at[t]] = [_table(r["table"], state["rows"][at[t]]), r["id_map"], int(r["rows"])]
        return out
    out = []
    for i, (q, elab) in enumerate(state["q"]):
        m = G.match(dg, q, cap=c["cap"] or None, order=order, model=model, count_only=kind == "count",
                    work_cap=c["work_cap"], directed=bool(c.get("directed")), edge_labels=elab)
        r = [m.count, m.id_map, m.pos2id, m.capped]
        if kind == "match":
            r.append(_table(m.rows, state["rows"][i]))
        out.append(r)
    return out


def work(case):
    """Bytes that any method has to touch. A query edge with labels (a, b) needs the data edges between those
    labels once: 2 m p(a) p(b) neighbour ids; the walks visit labels about as often as the data graph holds them,
    so p(a) p(b) is taken at its mean. Rows that come back count at the cap (their number is the query's own)."""
    kind = case["kind"]
    if kind == "grad":
        n = case["samples"]
        return {"bytes": 68 * n + 8 * 5313, "flops": 6 * 5248 * n}
    if kind == "build":
        return {"bytes": 16 * case["m"] + 8 * case["n"] + 4, "flops": 0}
    p = 1.0 / np.arange(1, case["labels"] + 1) ** case["zipf"]
    p = p / p.sum()
    qn = (case["qlo"] + case["qhi"]) / 2
    per_edge = 2 * case["m"] * float((p * p).sum()) * 4
    rows = min(case["cap"] or 2000, 200_000) * qn * 4 if kind in ("match", "serve") else 0
    return {"bytes": case["queries"] * ((qn - 1) * per_edge + rows), "flops": 0}


def exact(case, seed):
    """Loss and gradient in 64 bits (weights as the model holds them: bfloat16, biases in 32 bits). Every other
    case returns whole numbers, which have to be equal."""
    if case["kind"] != "grad":
        return None
    P = _Params(case, seed)
    h, f = 64, 16
    cut = np.cumsum([h * f, h, h * h, h, h, 1])
    w1, b1, w2, b2, w3, b3 = np.split(P.w, cut[:-1])
    half = lambda w: torch.from_numpy(w).bfloat16().double()  # noqa: E731
    w1, w2, w3 = half(w1).view(h, f), half(w2).view(h, h), half(w3)
    b1, b2, b3 = (torch.from_numpy(b).double() for b in (b1, b2, b3))
    x, y = torch.from_numpy(P.x).double(), torch.from_numpy(P.y).double()
    h1 = torch.relu(x @ w1.T + b1)
    h2 = torch.relu(h1 @ w2.T + b2)
    d = (h2 @ w3 + b3 - y) / len(y)
    loss = 0.5 * float((d * d).sum()) * len(y)
    d2 = d[:, None] * w3 * (h2 > 0)
    d1 = (d2 @ w2) * (h1 > 0)
    grad = torch.cat([(d1.T @ x).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), d @ h2, d.sum()[None]])
    return {"loss": loss, "grad": grad}
