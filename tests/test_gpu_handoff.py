"""GPU tests of the enumeration kernels' work handoff: queries whose root tasks
are far fewer than the GPU's warps and whose candidate-edge lists are mostly
shorter than a 32-entry chunk, so that nearly all of the search runs on warps
that were handed a part of a chunk's survivors.  Counts, local counts and
embeddings are compared with the CPU oracle, under several matching orders
(which move the levels that are split and the closed-form tail)."""
import os

import numpy as np
import pytest

import asdmatch_b200 as A
import oracle_util as O
from asdmatch_b200 import workloads as W
from test_zz_no_alloc import _count_noalloc

pytestmark = pytest.mark.gpu

CASES = [(5, 5252), (6, 5264), (7, 5270), (7, 5273), (8, 5281), (8, 5283), (8, 5289)]


@pytest.fixture(scope="module")
def dense(c0d_files):
    g, dpath, _ = c0d_files
    dg = A.DeviceGraph(g)
    yield g, dpath, dg
    dg.close()


def _connected_orders(q, cs, rng, count):
    """Orders that grow connected from the smallest candidate sets and from random vertices."""
    nbrs = [q.nbrs[q.offsets[u]:q.offsets[u + 1]].tolist() for u in range(q.n)]
    starts = np.argsort(cs.sizes())[:2].tolist() + rng.integers(0, q.n, count).tolist()
    for s in starts:
        order = [int(s)]
        while len(order) < q.n:
            order.append(int(rng.choice([w for u in order for w in nbrs[u] if w not in order])))
        yield order


@pytest.mark.parametrize("size,seed", CASES)
def test_handoff_counts(dense, workdir, size, seed):
    g, dpath, dg = dense
    q = g.random_walk_query(size, seed)
    qp = os.path.join(workdir, "handoff_%d.graph" % seed)
    q.write(qp)
    want, _ = O.oracle_run(qp, dpath)
    cs = A.CandidateSpace(dg, q)
    for order in _connected_orders(q, cs, np.random.default_rng(seed), 4):
        assert _count_noalloc(cs, A.Plan(cs, order)) == want, order
    cs.close()
    # the same query many times over in one launch: warps hand work of different queries to each other
    counts, status = A.run_batch(dg, [q] * 40)
    assert (status == A.OK).all() and (counts == want).all()


@pytest.mark.parametrize("size,seed", CASES[:4])
def test_handoff_local_and_embeddings(dense, workdir, size, seed):
    g, dpath, dg = dense
    q = g.random_walk_query(size, seed)
    qp, csv, emb = (os.path.join(workdir, "handoff_le_%d.%s" % (seed, x)) for x in ("graph", "csv", "emb"))
    q.write(qp)
    want, _ = O.oracle_run(qp, dpath, O.MODE_LOCAL, csv=csv)
    cs = A.CandidateSpace(dg, q)
    local = np.loadtxt(csv, delimiter=",", dtype=np.uint64, ndmin=2)
    for order in _connected_orders(q, cs, np.random.default_rng(seed), 1):
        plan = A.Plan(cs, order)
        r = A.adaptive_share_join(cs, plan, A.MODE_LOCAL)
        assert r.count == want and np.array_equal(r.local_counts, local)
        e = A.adaptive_share_join(cs, plan, A.MODE_EMBED, emb_capacity=want)
        rows = e.embeddings
        assert e.count == want and len(rows) == want
        # strictly ascending rows that are matches: each column's occurrences are the local counts
        prev, cur = rows[:-1], rows[1:]
        diff = cur != prev
        first = diff.argmax(1)
        at = np.arange(len(first))
        assert diff.any(1).all() and (cur[at, first] > prev[at, first]).all()
        for u in range(q.n):
            assert np.array_equal(np.bincount(rows[:, u], minlength=g.n).astype(np.uint64), local[:, u])
    cs.close()
