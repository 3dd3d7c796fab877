"""The filter's branches against the restated reference pipeline: label masks
of one and several words, graphs with too many labels for masks and for label
runs, and hubs whose runs a block scans (more of them in one chunk than its
list holds). Candidate sets, candidate-edge sizes and orders are whole
numbers and have to be equal; embeddings equal the restated joins' rows."""
import numpy as np
import pytest

import oracle
from gpsm_b200 import workloads as W
from test_parity_gpu import check_filter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,labels", [
    (4_096, 60_000, 1),      # one label: runs are whole lists
    (4_096, 60_000, 64),     # the last label of a one-word mask
    (4_096, 60_000, 65),     # the first of a second word
    (4_096, 60_000, 256),    # a full four-word mask
    (4_096, 60_000, 257),    # no masks: the directory is searched
    (33, 200, 3),            # less than one chunk of words
    (70_000, 300_000, 70_000),  # vertex and label bits exceed a key: no runs at all
])
@pytest.mark.parametrize("starts", [True, False])  # the table of starts, or masks and directory
def test_label_masks_and_their_absence(gpu, monkeypatch, n, m, labels, starts):
    monkeypatch.setenv("GPSM_DEBUG_NO_LABEL_STARTS", "0" if starts else "1")
    rng = np.random.default_rng(n + labels)
    e = rng.integers(0, n, (m, 2)) ** 2 // n  # low ids are popular: a skewed graph
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    lab = rng.permutation(np.arange(n) % labels) + 1
    g = W.graph_from_edges(n, e, lab)
    dg = gpu.DeviceGraph(g)
    for seed, (qn, mode) in enumerate([(3, W.MODE_TREE), (5, W.MODE_TREE), (5, W.MODE_DENSE), (6, W.MODE_INDUCED)]):
        q = W.random_walk_query(g, qn, seed, mode, 0.5)
        plan, d = check_filter(gpu, dg, g, q)
        if d["empty"]:
            continue
        ref, cnt, _, _ = plan.join(injective=True, cap=500)
        out = gpu.match(dg, q, cap=500)
        assert np.array_equal(out.rows, ref[:500])
    dg.free()


@pytest.mark.parametrize("hubs,leaves", [(5, 1023), (5, 1040), (100, 1500)])
def test_hubs_scanned_by_a_block(gpu, hubs, leaves):
    """Hub h (label 1) has `leaves` neighbours of label 2; only its last one
    goes on: to label 3 for even hubs, to label 5 for odd ones. One label-4
    neighbour each keeps hubs in the refinement."""
    edges, lab = [], [1] * hubs
    for h in range(hubs):
        for k in range(leaves):
            edges.append((h, len(lab)))
            lab.append(2)
        edges.append((len(lab) - 1, len(lab)))
        lab.append(3 if h % 2 == 0 else 5)
        edges.append((h, len(lab)))
        lab.append(4)
    g = W.graph_from_edges(len(lab), np.array(edges, np.uint32), np.array(lab, np.uint32))
    dg = gpu.DeviceGraph(g)
    for ql, qe in (([4, 1, 2, 3], [(0, 1), (1, 2), (2, 3)]), ([3, 2, 1, 4], [(0, 1), (1, 2), (2, 3)]),
                   ([2, 1, 2, 3], [(0, 1), (1, 2), (2, 3)])):
        q = W.Query(np.array(ql, np.uint32), np.array(qe, np.uint32))
        plan, d = check_filter(gpu, dg, g, q)
        assert not d["empty"]
        _, cnt = oracle.enumerate_embeddings(g, q, rows=False)
        assert gpu.match(dg, q, count_only=True).count == cnt
    dg.free()


@pytest.mark.parametrize("hubs,leaves", [
    (3, 7), (3, 8), (3, 9),      # the neighbours a pair's thread looks at, and one more
    (3, 39), (3, 40), (3, 41),   # and the first ones of the eight lanes after it
    (3, 128), (3, 129),          # runs a warp shares, runs in pieces
    (3, 256), (3, 257),          # one piece, two
    (700, 200),                  # more long runs and more pairs in a chunk than one pass takes
    (3, 4096), (3, 4097),        # the eight lanes, the whole block
    (40, 4200),                  # more of the latter than one pass lists
])
def test_run_lengths_where_the_split_changes(gpu, monkeypatch, hubs, leaves):
    """Hubs of label 1 at the lowest ids with `leaves` neighbours of label 2
    each, of which the last has a neighbour of label 3 (5 for odd hubs)."""
    monkeypatch.setenv("GPSM_DEBUG_NO_SMALL", "1")
    h = np.arange(hubs)
    first = hubs + h * leaves
    ends = hubs + hubs * leaves + h
    e = np.concatenate([
        np.stack([np.repeat(h, leaves), hubs + np.arange(hubs * leaves)], 1),
        np.stack([first + leaves - 1, ends], 1),
        np.stack([h, ends + hubs], 1)])
    lab = np.concatenate([np.full(hubs, 1), np.full(hubs * leaves, 2), np.where(h % 2 == 0, 3, 5), np.full(hubs, 4)])
    g = W.graph_from_edges(len(lab), e.astype(np.uint32), lab.astype(np.uint32))
    dg = gpu.DeviceGraph(g)
    for ql, qe in (([4, 1, 2, 3], [(0, 1), (1, 2), (2, 3)]), ([3, 2, 1, 4], [(0, 1), (1, 2), (2, 3)]),
                   ([1, 2, 2, 4], [(0, 1), (0, 2), (0, 3)])):
        check_filter(gpu, dg, g, W.Query(np.array(ql, np.uint32), np.array(qe, np.uint32)))
    dg.free()
