"""Small queries on small graphs run in one block (filter and join); with
GPSM_DEBUG_NO_SMALL=1 the general path takes them. Candidate counts, sizes,
orders, rows and join statistics have to be the same, at the sizes where the
two paths meet: tables at and past what the block holds, graphs at the limits
of vertices and entries, caps at, below and above the number of rows."""
import numpy as np
import pytest

from gpsm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _both(monkeypatch, f):
    monkeypatch.setenv("GPSM_DEBUG_NO_SMALL", "0")
    a = f()
    monkeypatch.setenv("GPSM_DEBUG_NO_SMALL", "1")
    return a, f()


def _same(gpu, dg, q, monkeypatch, **kw):
    def run():
        out = gpu.match(dg, q, **kw)
        return out, [x.copy() for x in gpu.last_levels(q.n)], gpu.debug_filter(dg, q, with_candidates=True)
    (a, la, fa), (b, lb, fb) = _both(monkeypatch, run)
    assert fa["empty"] == fb["empty"]
    for k in ("cand_count", "size_fwd", "size_rev", "filter_order", "plain_pos2id", "candidates"):
        assert np.array_equal(fa[k], fb[k]), k
    assert a.count == b.count and a.capped == b.capped
    assert np.array_equal(a.id_map, b.id_map) and np.array_equal(a.pos2id, b.pos2id)
    assert np.array_equal(a.rows, b.rows)
    assert a.info["cands_scanned"] == b.info["cands_scanned"]
    for x, y in zip(la, lb):
        assert np.array_equal(x, y)
    return a


@pytest.mark.parametrize("n,m,labels", [
    (40, 100, 2),            # a few words
    (2_000, 12_000, 3),      # tables past the block's: the general join takes over
    (10_000, 40_000, 8),
    (32_768, 199_999, 30),   # the most vertices
    (32_769, 100_000, 30),   # one vertex too many: the general path twice
    (9_000, 200_000, 40),    # the most entries
])
@pytest.mark.parametrize("skew", [False, True])
def test_same_results_as_the_general_path(gpu, monkeypatch, n, m, labels, skew):
    rng = np.random.default_rng(n + labels)
    e = rng.integers(0, n, (m, 2))
    if skew:
        e[:, 0] = e[:, 0] ** 3 // n ** 2  # hubs among the low ids
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    g = W.graph_from_edges(n, e, (rng.integers(0, labels, n) + 1).astype(np.uint32))
    dg = gpu.DeviceGraph(g)
    model = gpu.Model(0, seed=4)
    seen = 0
    for seed, (qn, mode) in enumerate([(2, W.MODE_TREE), (3, W.MODE_TREE), (5, W.MODE_TREE), (5, W.MODE_DENSE),
                                       (8, W.MODE_TREE), (8, W.MODE_INDUCED)]):
        q = W.random_walk_query(g, qn, 31 * seed + n, mode, 0.4)
        a = _same(gpu, dg, q, monkeypatch, cap=200_000, work_cap=1 << 28)
        seen += a.count
        _same(gpu, dg, q, monkeypatch, cap=200_000, work_cap=1 << 28, order="learned", model=model)
        for cap in {1, max(a.count - 1, 1), max(a.count, 1), a.count + 1}:
            x, y = _both(monkeypatch, lambda: gpu.match(dg, q, cap=cap, work_cap=1 << 28))
            assert x.count == y.count and x.capped == y.capped and np.array_equal(x.rows, y.rows)
            assert np.array_equal(x.rows[: a.count], a.rows[:cap])
    assert seen > 0
    dg.free()


def test_no_match_and_absent_labels(gpu, monkeypatch):
    g = W.graph_from_edges(6, np.array([[0, 1], [2, 3], [4, 5]]), np.array([1, 2, 2, 3, 1, 3], np.uint32))
    dg = gpu.DeviceGraph(g)
    for ql, qe in (([1, 2, 3], [(0, 1), (1, 2)]), ([1, 9], [(0, 1)]), ([1, 2], [(0, 1)])):
        q = W.Query(np.array(ql, np.uint32), np.array(qe, np.uint32))
        a, b = _both(monkeypatch, lambda: gpu.match(dg, q))
        assert a.count == b.count and a.empty_filter == b.empty_filter and np.array_equal(a.rows, b.rows)
    assert a.count == 1


def test_batches_of_both_paths(gpu, monkeypatch, small_er):
    dg = gpu.DeviceGraph(small_er.graph)
    qs = [W.random_walk_query(small_er.graph, 3 + k % 6, k, W.MODE_TREE) for k in range(40)]
    for slots in (1, 4):
        a, b = _both(monkeypatch, lambda: gpu.match_batch(dg, qs, slots=slots, slot_arena=1 << 30 if slots > 1 else 0))
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    dg.free()
