"""Directed, labelled queries: testing each edge in the step that completes it
(no work cap) gives exactly the rows that verifying finished rows gives (the
path of queries with a work cap), in the same order, with the edge table and
with list searches, complete and cut by an embedding cap."""
import numpy as np
import pytest

from gpsm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [True, False])
@pytest.mark.parametrize("qn,mode", [(2, W.MODE_TREE), (4, W.MODE_TREE), (4, W.MODE_DENSE), (6, W.MODE_INDUCED)])
def test_edge_tests_in_the_steps_equal_verified_rows(gpu, monkeypatch, qn, mode, table):
    monkeypatch.setenv("GPSM_DEBUG_NO_EDGE_HASH", "0" if table else "1")
    g = W.rmat_graph(11, 20_000, 6, 0.5, seed=21)
    dg = gpu.DeviceGraph(g)
    rng = np.random.default_rng(3)
    back = rng.random(g.m) < 0.5
    lab = rng.integers(1, 3, g.m).astype(np.uint32)
    both = rng.random(g.m) < 0.3  # some pairs in both directions, the second with label 1
    e = np.where(back[:, None], g.edges[:, ::-1], g.edges)
    dg.set_directed(np.concatenate([e, e[both][:, ::-1]]), np.concatenate([lab, np.ones(both.sum(), np.uint32)]))
    kind = {(int(a), int(b)): int(x) for (a, b), x in zip(e, lab)}
    kept = 0
    for seed in range(4):
        q = W.random_walk_query(g, qn, seed, mode, 0.5)
        a, b = q.data_ids[q.edges[:, 0]], q.data_ids[q.edges[:, 1]]
        turn = np.array([(int(x), int(y)) not in kind for x, y in zip(a, b)])
        q.edges = np.ascontiguousarray(np.where(turn[:, None], q.edges[:, ::-1], q.edges))
        el = np.array([kind[(int(q.data_ids[x]), int(q.data_ids[y]))] for x, y in q.edges], np.uint32)
        got = gpu.match(dg, q, directed=True, edge_labels=el)
        want = gpu.match(dg, q, directed=True, edge_labels=el, work_cap=10**12)
        assert not want.info["aborted"]
        assert np.array_equal(got.rows, want.rows)
        kept += got.count
        for cap in (1, 37, 20_000):
            cut = gpu.match(dg, q, cap=cap, directed=True, edge_labels=el)
            assert cut.capped == (got.count >= cap)
            assert np.array_equal(cut.rows, got.rows[:cap])
    assert kept > 0
    dg.free()
