"""GPU test of the local-count matrices' way to the caller: large matrices,
mostly candidates (copied whole) and mostly not (gathered and scattered), into
buffers that hold other values before the call, alone and batched, with an
empty query among them.  Expected values are closed forms over the degrees."""
import ctypes as C

import numpy as np
import pytest

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu


def _graph(n, m, labels, seed):
    rng = np.random.default_rng(seed)
    e = np.unique(np.sort(rng.integers(0, n, (m, 2)), 1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    lab = rng.integers(0, labels, n)
    return A.HostGraph.from_edges(n, lab, e), lab, e


def _star(lab, e, n, centre, leaves):
    """Local counts of the query centre - leaf (two leaves of one label each): columns (centre, leaf, leaf)."""
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    d = np.bincount(src[lab[dst] == leaves], minlength=n).astype(np.int64)  # neighbours of the leaves' label
    mid = np.where(lab == centre, d * (d - 1), 0)
    use = (lab[src] == leaves) & (lab[dst] == centre)
    end = np.zeros(n, np.int64)
    np.add.at(end, src[use], d[dst[use]] - 1)
    return np.stack([mid, end, end], 1).astype(np.uint64)


@pytest.mark.parametrize("n,m,labels", [(2000, 9000, 1), (420_000, 900_000, 1), (420_000, 900_000, 7)])
def test_matrices(n, m, labels):
    g, lab, e = _graph(n, m, labels, n + labels)
    centre, leaves = 0, min(1, labels - 1)
    want = _star(lab, e, n, centre, leaves)
    q = A.HostGraph.from_edges(3, [centre, leaves, leaves], [[0, 1], [0, 2]])
    none = A.HostGraph.from_edges(2, [labels + 3, 0], [[0, 1]])  # a label the graph does not have
    dg = A.DeviceGraph(g)
    cs = A.CandidateSpace(dg, q)
    plan = A.Plan(cs, [1, 0, 2])
    got = np.full((n, 3), 7, np.uint64)
    opts, st = A.RunOpts(), A.RunStats()
    opts.mode, opts.local_counts = A.MODE_LOCAL, A._ptr(got, A._u64p)
    assert A._run_plan(cs._h, plan._h, C.byref(opts), C.byref(st)) == A.OK
    assert st.count == want[:, 0].sum() and np.array_equal(got, want)
    cs.close()
    b = A.BatchInput([q, none, q])
    mats = [np.full((n, k), 9, np.uint64) for k in (3, 2, 3)]
    ptrs = (A._u64p * 3)(*[A._ptr(x, A._u64p) for x in mats])
    rc = A._run_batch_local(dg._h, 3, A._ptr(b.sizes), A._ptr(b.ob, A._u64p), A._ptr(b.offs), A._ptr(b.nb, A._u64p),
                            A._ptr(b.nbrs), A._ptr(b.lb, A._u64p), A._ptr(b.labs), 0.0, A._ptr(b.counts, A._u64p),
                            b.status.ctypes.data_as(C.POINTER(C.c_int)), ptrs, C.byref(st))
    assert rc == A.OK and b.counts.tolist() == [st.count // 2, 0, st.count // 2]
    assert np.array_equal(mats[0], want) and np.array_equal(mats[2], want) and not mats[1].any()
    dg.close()
