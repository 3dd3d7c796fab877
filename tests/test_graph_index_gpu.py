"""The device-built label index at its edges: one vertex, no edges, isolated
vertices at either end of the id range, label values too large for a rank
table, hubs, and the two ways to make a graph (host CSR, edge list) giving
the same matches and candidate sets as the restated reference pipeline."""
import numpy as np
import pytest

from gpsm_b200 import GpsmError
from gpsm_b200 import workloads as W
from test_parity_gpu import check_filter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,labels,spread", [
    (1, 0, 1, 1),            # a single vertex
    (300, 0, 4, 1),          # no edges
    (300, 40, 4, 1),         # mostly isolated vertices
    (5_000, 30_000, 7, 1),
    (5_000, 30_000, 7, 700_000_001),  # label values past the rank table
    (2_049, 2_048, 3, 1),    # a star: one hub with every entry of a tile and one more
])
def test_index_of_both_builds(gpu, n, m, labels, spread):
    rng = np.random.default_rng(n + m)
    if m == n - 1:
        e = np.stack([np.zeros(m, np.int64), np.arange(1, n)], 1)
    else:
        e = rng.integers(n // 10, max(n - n // 10, 1), (m, 2))
        e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    lab = (rng.integers(0, labels, n) * spread + 1).astype(np.uint32)
    g = W.graph_from_edges(n, e, lab)
    both = [gpu.DeviceGraph(g), gpu.DeviceGraph(g, build_on_device=True)]
    for dg in both:
        off, cols = dg.download()
        assert np.array_equal(off, g.offsets) and np.array_equal(cols, g.cols)
        one = gpu.match(dg, W.Query(lab[:1].copy(), np.zeros((0, 2), np.uint32)))
        assert np.array_equal(np.sort(one.rows[:, 0]), np.flatnonzero(lab == lab[0]))
        if g.m > 10:
            for seed, mode in enumerate([W.MODE_TREE, W.MODE_DENSE]):
                check_filter(gpu, dg, g, W.random_walk_query(g, 3, seed, mode, 0.5))
        dg.free()


def test_an_edge_to_no_vertex_is_refused(gpu):
    g = W.graph_from_edges(10, np.array([[0, 1], [2, 3]]), np.ones(10, np.uint32))
    g.edges = np.array([[0, 1], [2, 10]], np.uint32)
    with pytest.raises(GpsmError) as err:
        gpu.DeviceGraph(g, build_on_device=True)
    assert err.value.code == -1  # GPSM_ERR_INVALID
