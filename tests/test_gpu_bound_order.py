"""GPU test of the overflow proofs' two forms: with the bound's value asked for
(every bound of every query runs) and, in the counting entry points, without
(cheapest bound first, queries that an upper bound keeps below 2^64 dropped).
Both have to prove the same queries, and a query that is dropped must have a
lower bound below 2^64."""
import numpy as np
import pytest

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu

SHAPES = [(3000, 12000, 3, 1), (60_000, 300_000, 8, 2), (60_000, 300_000, 20, 3), (200_000, 900_000, 2, 4)]


@pytest.mark.parametrize("n,m,labels,seed", SHAPES)
def test_proofs_agree(n, m, labels, seed):
    g = A.HostGraph.chung_lu(n, m, 2.1, labels, 1.0, seed)
    dg = A.DeviceGraph(g)
    qs = [g.random_walk_query(size, 100 * seed + 7 * size + i) for size in (2, 3, 6, 9, 12, 16, 20, 26, 32)
          for i in range(3)]
    b = A.BatchInput(qs)
    A.run_batch_ex(dg, b, count_limit=10 ** 7, query_time_limit_s=0.01)
    for q, st in zip(qs, b.status):
        cs = A.CandidateSpace(dg, q)
        lower, exceeds = cs.count_lower_bound()
        cs.close()
        assert exceeds == (lower == 2 ** 64 - 1)
        assert (st == A.ERR_OVERFLOW) == exceeds, (q.n, lower, st)
    dg.close()


def test_single_query_agrees():
    g = A.HostGraph.chung_lu(60_000, 300_000, 2.1, 4, 1.0, 9)
    dg = A.DeviceGraph(g)
    for size in (5, 14, 24, 32):
        q = g.random_walk_query(size, 31 * size)
        cs = A.CandidateSpace(dg, q)
        _, exceeds = cs.count_lower_bound()
        try:
            A.adaptive_share_join(cs, count_limit=10 ** 7, time_limit_s=0.5)
            code = A.OK
        except A.AsdmError as e:
            code = e.code
        cs.close()
        assert (code == A.ERR_OVERFLOW) == exceeds
    dg.close()
