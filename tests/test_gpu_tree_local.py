"""GPU test of the tree program's local counts by inclusion-exclusion: trees
whose same-label vertices are siblings, cousins' parents, or both, up to four
of one label, against the CPU oracle's LOCAL_COUNT matrix, alone and batched."""
import os

import numpy as np
import pytest

import asdmatch_b200 as A
import oracle_util as O

pytestmark = pytest.mark.gpu

TREES = {  # labels, edges
    "star3": ([0, 1, 1, 1], [[0, 1], [0, 2], [0, 3]]),
    "star4_one_label": ([0, 0, 0, 0, 0], [[0, 1], [0, 2], [0, 3], [0, 4]]),
    "grandparent": ([1, 0, 1], [[0, 1], [1, 2]]),
    "path_with_siblings": ([0, 1, 0, 2, 2], [[0, 1], [1, 2], [2, 3], [2, 4]]),
    "two_stars": ([0, 1, 1, 2, 2, 3], [[0, 1], [0, 2], [0, 5], [5, 3], [5, 4]]),
    "leaf_and_inner": ([0, 1, 2, 1, 3], [[0, 1], [0, 3], [1, 2], [3, 4]]),
    "far_pair": ([0, 1, 2, 0], [[0, 1], [1, 2], [2, 3]]),  # closes a cycle when merged: enumerated
    "no_conflict": ([0, 1, 2, 3], [[0, 1], [1, 2], [2, 3]]),
}


@pytest.mark.parametrize("n,m,labels,seed", [(60, 150, 4, 1), (400, 1500, 4, 2), (3000, 9000, 5, 3)])
def test_tree_local_counts(workdir, n, m, labels, seed):
    rng = np.random.default_rng(seed)
    e = np.unique(np.sort(np.minimum(rng.integers(0, n, (m, 2)), rng.integers(0, n, (m, 2))), 1), axis=0)  # uneven degrees
    e = e[e[:, 0] != e[:, 1]]
    g = A.HostGraph.from_edges(n, rng.integers(0, labels, n), e)
    d = os.path.join(workdir, "treelocal%d" % seed)
    os.makedirs(d)
    dpath, qpath, csv = (os.path.join(d, x) for x in ("data", "query", "csv"))
    g.write(dpath)
    dg = A.DeviceGraph(g)
    qs, want = [], []
    for lab, edges in TREES.values():
        q = A.HostGraph.from_edges(len(lab), lab, edges)
        q.write(qpath)
        count, _ = O.oracle_run(qpath, dpath, O.MODE_LOCAL, csv=csv)
        local = np.loadtxt(csv, delimiter=",", dtype=np.uint64, ndmin=2)
        r = A.match(dg, q, A.MODE_LOCAL)
        assert r.count == count and np.array_equal(r.local_counts, local)
        qs.append(q)
        want.append((count, local))
    counts, status, local = A.run_batch_local(dg, qs)
    for (c, l), got, st, m2 in zip(want, counts, status, local):
        assert st == A.OK and got == c and np.array_equal(m2, l)
    dg.close()
