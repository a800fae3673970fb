"""GPU test of trees with same-label vertices three or more edges apart in LOCAL
mode: queries with many matches are counted as maps that are injective around
every vertex, less the embeddings of the quotients that merge such vertices.
Whole numbers, so equal: to the CPU oracle's LOCAL_COUNT matrix on a small
graph, and on a dense one to the enumeration of the query itself, which a run
with a time limit takes."""
import os

import numpy as np
import pytest

import asdmatch_b200 as A
import oracle_util as O

pytestmark = pytest.mark.gpu


def path(n):
    return [[i, i + 1] for i in range(n - 1)]


TREES = {  # labels, edges
    "ends": ([0, 1, 2, 0, 3], path(4) + [[3, 4]]),                     # closes a triangle, a leaf beside it
    "ends4": ([0, 1, 2, 1, 0], path(5)),                               # a near pair inside, a 4-cycle
    "ends5": ([0, 1, 2, 3, 1, 0], path(6)),                            # two far pairs, four and five edges apart
    "adjacent_copy": ([0, 1, 2, 0, 0], path(5)),                       # the far vertex joins either of two neighbours
    "two_pairs": ([0, 1, 2, 0, 1], path(5)),                           # three quotients: one pair, the other, both
    "near_at_far": ([0, 0, 1, 2, 0], [[0, 2], [1, 2], [2, 3], [3, 4]]),  # the far vertex joins either sibling
    "branch": ([0, 1, 2, 0, 3], path(4) + [[1, 4]]),                   # a branch at the cycle
    "near_chain": ([0, 1, 0, 1, 0], path(5)),                          # ends far, each near to the middle
    "one_label": ([0, 0, 0, 0, 0], path(5)),                           # near and far pairs of one label
    "claw": ([0, 1, 2, 1, 3, 1], [[0, 1], [0, 2], [0, 4], [2, 3], [4, 5]]),  # three of a label, pairwise far
    "near_far_claw": ([0, 1, 2, 1, 1], [[0, 1], [0, 2], [2, 3], [2, 4]]),  # a far vertex beside two near ones
}


def graph(n, m, seed):
    rng = np.random.default_rng(seed)
    e = np.unique(np.sort(np.minimum(rng.integers(0, n, (m, 2)), rng.integers(0, n, (m, 2))), 1), axis=0)  # uneven degrees
    return A.HostGraph.from_edges(n, rng.integers(0, 4, n), e[e[:, 0] != e[:, 1]])


def test_oracle(workdir):
    g = graph(150, 4000, 1)
    d = os.path.join(workdir, "far")
    os.makedirs(d)
    dpath, qpath, csv = (os.path.join(d, x) for x in ("data", "query", "csv"))
    g.write(dpath)
    dg = A.DeviceGraph(g)
    for lab, edges in TREES.values():
        q = A.HostGraph.from_edges(len(lab), lab, edges)
        q.write(qpath)
        count, _ = O.oracle_run(qpath, dpath, O.MODE_LOCAL, csv=csv)
        r = A.match(dg, q, A.MODE_LOCAL)
        assert r.count == count
        assert np.array_equal(r.local_counts, np.loadtxt(csv, delimiter=",", dtype=np.uint64, ndmin=2))
    dg.close()


def test_quotients_equal_enumeration():
    dg = A.DeviceGraph(graph(2500, 250_000, 2))
    qs = [A.HostGraph.from_edges(len(lab), lab, edges) for lab, edges in TREES.values()]
    for q, name in zip(qs, TREES):
        limited, free = A.match(dg, q, A.MODE_LOCAL, time_limit_s=300.0), A.match(dg, q, A.MODE_LOCAL)
        assert limited.count > 2 ** 29 and limited.count == free.count, name
        assert np.array_equal(limited.local_counts, free.local_counts), name
        assert free.list_bytes != limited.list_bytes, name  # (the quotients ran)
    counts, status, local = A.run_batch_local(dg, qs)
    want, wstatus, wlocal = A.run_batch_local(dg, qs, 300.0)
    assert np.array_equal(counts, want) and not status.any() and not wstatus.any()
    assert all(np.array_equal(a, b) for a, b in zip(local, wlocal))
    dg.close()
