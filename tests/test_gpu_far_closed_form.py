"""GPU test of LOCAL mode's counts through quotients (trees with same-label
vertices three or more edges apart) against sums over partitions in numpy: the
embeddings are the homomorphisms of every quotient by blocks of non-adjacent
same-label vertices, with the partition lattice's signs, and each quotient's
homomorphisms are a contraction of the 0/1 adjacency matrix.  Every value is a
whole number below 2^53, so float64 contractions are exact."""
import math

import numpy as np
import pytest

import asdmatch_b200 as A
from test_gpu_far_pairs import TREES

pytestmark = pytest.mark.gpu

PER_LABEL = 80  # 80^5 maps and more at this density: past the rule's sizes


@pytest.fixture(scope="module")
def data():
    rng = np.random.default_rng(7)
    n = 4 * PER_LABEL
    adj = np.triu(rng.random((n, n)) < 0.9, 1)
    adj = adj | adj.T
    labels = rng.permutation(np.repeat(np.arange(4), PER_LABEL))
    dg = A.DeviceGraph(A.HostGraph.from_edges(n, labels, np.argwhere(np.triu(adj))))
    yield labels, adj.astype(np.float64), dg
    dg.close()


def _partitions(lab, edges):
    """Partitions of the vertices into blocks of one label without an edge inside."""
    joined = {frozenset(e) for e in map(tuple, edges)}

    def place(u, blocks):
        if u == len(lab):
            yield [list(b) for b in blocks]
            return
        for b in blocks:
            if lab[b[0]] == lab[u] and all(frozenset((u, w)) not in joined for w in b):
                b.append(u)
                yield from place(u + 1, blocks)
                b.pop()
        yield from place(u + 1, blocks + [[u]])
    return place(0, [])


def _local_counts(labels, adj, lab, edges):
    out = np.zeros((len(labels), len(lab)))
    of = [np.nonzero(labels == k)[0] for k in range(4)]
    for blocks in _partitions(lab, edges):
        at = {u: b for b, members in enumerate(blocks) for u in members}
        sign = math.prod((-1) ** (len(b) - 1) * math.factorial(len(b) - 1) for b in blocks)
        args = []
        for x, y in sorted({tuple(sorted((at[u], at[w]))) for u, w in edges}):
            args += [adj[np.ix_(of[lab[blocks[x][0]]], of[lab[blocks[y][0]]])], [x, y]]
        for b, members in enumerate(blocks):
            homs = np.einsum(*args, [b], optimize="optimal")
            for u in members:
                out[of[lab[u]], u] += sign * homs
    return out


def test_quotients_equal_partition_sums(data):
    labels, adj, dg = data
    qs, want = [], []
    for lab, edges in TREES.values():
        qs.append(A.HostGraph.from_edges(len(lab), lab, edges))
        want.append(_local_counts(labels, adj, lab, edges))
        assert want[-1].max() < 2 ** 53
    for q, w, name in zip(qs, want, TREES):
        r = A.match(dg, q, A.MODE_LOCAL)
        assert r.count == int(w[:, 0].sum()) > 2 ** 29, name
        assert np.array_equal(r.local_counts, w.astype(np.uint64)), name
        assert r.intersections > 0, name  # the quotients were enumerated: a tree's own levels have one list each
    counts, status, local = A.run_batch_local(dg, qs)
    assert not status.any()
    for c, m, w in zip(counts, local, want):
        assert c == int(w[:, 0].sum()) and np.array_equal(m, w.astype(np.uint64))
