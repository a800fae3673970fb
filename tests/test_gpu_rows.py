"""GPU tests of the sorted embedding rows: packed keys of one and of several
words, row counts around the sort's tile and the host/device boundary, ties in
the first word, single-vertex queries.  Expected rows are written down with
numpy from graphs whose embeddings are known by construction."""
import numpy as np
import pytest

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu


def _permuted(rng, labels, edges):
    """The graph with its ids shuffled: (host graph, new id of each old id)."""
    n = len(labels)
    new = rng.permutation(n).astype(np.uint32)
    lab = np.zeros(n, np.uint32)
    lab[new] = labels
    return A.HostGraph.from_edges(n, lab, new[np.asarray(edges, np.int64)]), new


def _embeddings(g, q):
    dg = A.DeviceGraph(g)
    r = A.match(dg, q, A.MODE_EMBED)
    dg.close()
    return r.embeddings


def _sorted(rows):
    return rows[np.lexsort(rows.T[::-1])]


# rows = a * b: single rows, the host/device boundary (4096), tiles of 4096
@pytest.mark.parametrize("a,b", [(1, 1), (1, 7), (23, 89), (2, 1024), (683, 3), (5, 819), (3, 1365), (64, 64), (17, 241), (1366, 6),
                                 (300, 431), (65, 2050)])
def test_product_rows(a, b):
    rng = np.random.default_rng(a * 10_007 + b)
    labels = np.array([0] * a + [1] * b)
    edges = np.stack(np.meshgrid(np.arange(a), a + np.arange(b), indexing="ij"), -1).reshape(-1, 2)
    g, new = _permuted(rng, labels, edges)
    for order in ([0, 1], [1, 0]):
        q = A.HostGraph.from_edges(2, order, [[0, 1]])
        want = new[edges] if order == [0, 1] else new[edges[:, ::-1]]
        assert np.array_equal(_embeddings(g, q), _sorted(want))


def test_single_vertex_rows():
    rng = np.random.default_rng(4)
    labels = rng.integers(0, 3, 9000)
    edges = [[i, i + 1] for i in range(8999)]
    g, new = _permuted(rng, labels, edges)
    q = A.HostGraph.from_edges(1, [1], [])
    assert np.array_equal(_embeddings(g, q)[:, 0], np.sort(new[np.nonzero(labels == 1)[0]]))


@pytest.mark.parametrize("paths,first,second", [(40_000, 3, 2), (700, 2, 3), (33_000, 1, 1)])
def test_rows_of_several_words(paths, first, second):
    """Disjoint brooms: a path of four labels whose end has `first` leaves of one label and `second` of another.  The
    first word holds the path's four fields, so the leaves' rows tie in it."""
    rng = np.random.default_rng(paths)
    k = 4 + first + second
    base = np.arange(paths)[:, None] * k
    edges = [base + [[i, i + 1]] for i in range(3)] + [base + [[3, 4 + i]] for i in range(first + second)]
    labels = np.tile([0, 1, 2, 3] + [4] * first + [5] * second, paths)
    g, new = _permuted(rng, labels, np.concatenate(edges))
    q = A.HostGraph.from_edges(6, [0, 1, 2, 3, 4, 5], [[0, 1], [1, 2], [2, 3], [3, 4], [3, 5]])
    want = [np.concatenate([base + [[0, 1, 2, 3, 4 + i, 4 + first + j]]]) for i in range(first) for j in range(second)]
    assert np.array_equal(_embeddings(g, q), _sorted(new[np.concatenate(want)]))


def test_capacity_is_checked():
    labels = np.array([0] * 50 + [1] * 60)
    edges = [[i, 50 + j] for i in range(50) for j in range(60)]
    g = A.HostGraph.from_edges(110, labels, edges)
    dg = A.DeviceGraph(g)
    cs = A.CandidateSpace(dg, A.HostGraph.from_edges(2, [0, 1], [[0, 1]]))
    with pytest.raises(A.AsdmError) as e:
        A.adaptive_share_join(cs, mode=A.MODE_EMBED, emb_capacity=2999)
    assert e.value.code == A.ERR_CAPACITY
    assert len(A.adaptive_share_join(cs, mode=A.MODE_EMBED, emb_capacity=3000).embeddings) == 3000
    cs.close()
    dg.close()
