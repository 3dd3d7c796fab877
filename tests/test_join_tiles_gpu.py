"""Join steps over tiles of candidates: rows of one candidate and rows longer
than a tile, graphs with and without parallel edges (only the former look for
a neighbour listed twice), checks against no, one and several same-label
columns, by the edge table and by the lists. The small-query path is off, so
every row comes from the general one; the rows are the backtracking oracle's."""
import numpy as np
import pytest

import oracle
from gpsm_b200 import workloads as W
from test_parity_gpu import _graph

pytestmark = pytest.mark.gpu


def _random(n, m, labels, seed):
    rng = np.random.default_rng(seed)
    e = rng.integers(0, n, (m, 2))
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    return n, e, (rng.integers(0, labels, n) + 1).astype(np.uint32)


def _hub(n):
    """A hub with every vertex as a neighbour, and a path through them."""
    e = [(0, i) for i in range(1, n)] + [(i, i + 1) for i in range(1, n - 1)]
    return n, np.array(e), np.array([1] + [2] * (n - 1), np.uint32)


def _sorted(rows):
    return rows[np.lexsort(rows.T[::-1])]


GRAPHS = {
    "short": _random(4_000, 9_000, 6, 1),
    "one_label": _random(220, 700, 1, 2),
    "dense": _random(90, 1_800, 2, 3),
    "hub_under_a_tile": _hub(1_024),  # 1023 candidates in one row
    "hub_over_a_tile": _hub(1_026),   # 1025
    "hub_of_tiles": _hub(2_600),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("repeated", [False, True])
@pytest.mark.parametrize("lists", [False, True])
def test_rows_are_the_oracles(gpu, monkeypatch, name, repeated, lists):
    monkeypatch.setenv("GPSM_DEBUG_NO_SMALL", "1")
    monkeypatch.setenv("GPSM_DEBUG_NO_EDGE_HASH", "1" if lists else "0")
    n, e, lab = GRAPHS[name]
    g = W.graph_from_edges(n, e, lab)
    every_third = e[::3]
    dg = gpu.DeviceGraph(_graph(n, np.concatenate([e, every_third, every_third]).tolist(), lab) if repeated else g)
    q_hub = W.Query(np.array([1, 2, 2], np.uint32), np.array([[0, 1], [0, 2], [1, 2]], np.uint32))
    queries = [q_hub] if name.startswith("hub") else [
        W.random_walk_query(g, k, 5 * k, mode, 0.5) for k, mode in
        [(2, W.MODE_TREE), (3, W.MODE_TREE), (4, W.MODE_DENSE), (4, W.MODE_INDUCED)]]
    for q in queries:
        rows, cnt = oracle.enumerate_embeddings(g, q)
        out = gpu.match(dg, q, cap=1 << 22)
        assert out.count == cnt
        assert np.array_equal(_sorted(out.embeddings()), _sorted(np.asarray(rows, np.uint32).reshape(-1, q.n)))
    dg.free()


@pytest.mark.parametrize("every", [1, 3, 40])
def test_rows_found_past_tiles_without_rows(gpu, monkeypatch, every):
    """A level of 90,000 rows whose candidates are nearly all rejected: only
    every `every`-th vertex of A closes a triangle, with one vertex of B, so
    the kept rows lie up to 360 check tiles apart, and the next step finds
    them by their tiles' offsets."""
    monkeypatch.setenv("GPSM_DEBUG_NO_SMALL", "1")
    rng = np.random.default_rng(every)
    na, nb, nc = 300, 300, 900
    a, b, c, d = 0, na, na + nb, na + nb + nc  # first ids of the labels 1..4; c's first half and second half
    e = {(x, b + y) for x in range(na) for y in range(nb)}
    for x in range(na):  # A knows the first half, B the second
        e |= {(x, c + int(z)) for z in rng.choice(nc // 2, 30, replace=False)}
    for y in range(nb):
        e |= {(b + y, c + nc // 2 + int(z)) for z in rng.choice(nc // 2, 30, replace=False)}
    e |= {(x, c + nc // 2) for x in range(0, na, every)}  # but for one vertex of the other half
    e |= {(b, c + nc // 2)} | {(b + y, c) for y in range(1, nb)}
    e |= {(c + z, d + z) for z in range(nc)}
    lab = np.repeat(np.arange(1, 5), [na, nb, nc, nc]).astype(np.uint32)
    g = W.graph_from_edges(len(lab), np.array(sorted(e), np.uint32), lab)
    q = W.Query(np.array([1, 2, 3, 4], np.uint32), np.array([[0, 1], [0, 2], [1, 2], [2, 3]], np.uint32))
    rows, cnt = oracle.enumerate_embeddings(g, q)
    dg = gpu.DeviceGraph(g)
    for lists in ("0", "1"):
        monkeypatch.setenv("GPSM_DEBUG_NO_EDGE_HASH", lists)
        out = gpu.match(dg, q, order=[0, 1, 2, 3])
        assert out.count == cnt
        assert np.array_equal(_sorted(out.embeddings()), _sorted(np.asarray(rows, np.uint32).reshape(-1, 4)))
    dg.free()
