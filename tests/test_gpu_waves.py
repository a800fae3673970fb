"""GPU tests of the candidate-set waves (K1, K2) at the edges of a bitset word
and of the words per warp: label sizes around 32, one-label graphs, queries
whose waves are many, and the phantom vertex 0; compared with the CPU oracle's
candidate-space dump, alone and in a group."""
import os

import numpy as np
import pytest

import asdmatch_b200 as A
import oracle_util as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,labels,seed", [(6, 9, 1, 1), (31, 60, 1, 2), (32, 70, 1, 3), (33, 64, 1, 4), (64, 200, 2, 5),
                                             (65, 190, 2, 6), (97, 300, 3, 7), (1025, 3000, 1, 8), (2050, 6000, 2, 9),
                                             (3000, 9000, 64, 10)])
def test_candidate_spaces_match_the_oracle(workdir, n, m, labels, seed):
    rng = np.random.default_rng(seed)
    # a ring keeps the graph connected; vertex 0 has the most neighbours, so it often is the phantom's effect
    ring = {(i, i + 1) for i in range(n - 1)}
    hub = {(0, int(v)) for v in rng.integers(2, n, max(1, n // 8))}
    rest = {tuple(sorted(map(int, e))) for e in rng.integers(0, n, (2 * m, 2)) if e[0] != e[1]}
    edges = sorted(ring | hub | set(sorted(rest)[:m]))
    g = A.HostGraph.from_edges(n, rng.integers(0, labels, n), edges)
    d = os.path.join(workdir, "waves%d" % seed)
    os.makedirs(d)
    dpath, qpath, cpath = (os.path.join(d, x) for x in ("data", "query", "cs"))
    g.write(dpath)
    dg = A.DeviceGraph(g)
    qs, want = [], []
    for size in (2, 3, 5, min(7, n)) if n < 100 else (2, 3, 4):  # (the oracle also counts the matches)
        q = g.random_walk_query(size, 50 * seed + size)
        q.write(qpath)
        O.oracle_run(qpath, dpath, cs=cpath)
        qs.append(q)
        want.append(open(cpath).read())
    group = A.candidate_spaces(dg, qs)
    for q, w, cs in zip(qs, want, group):
        assert cs.write_to_stream() == w
        alone = A.CandidateSpace(dg, q)
        assert alone.write_to_stream() == w
        alone.close()
        cs.close()
    dg.close()
