"""GPU test of where an estimator's memory lies: beside the pool that calls take
their scratch from (the device's current pool), whose large blocks a lasting
one would break up, and given back when estimators are freed."""
import gc

import numpy as np
import pytest

import asdmatch_b200 as A
from test_zz_no_alloc import _PoolWatch

pytestmark = pytest.mark.gpu


def _batch(graphs):
    """`graphs` triangles."""
    n = 3 * graphs
    v = np.arange(n)
    adj = (v[:, None] // 3 * 3 + (v[:, None] + [[1, 2]]) % 3).astype(np.uint32)
    x = np.random.default_rng(graphs).uniform(-1, 1, (n, 44)).astype(np.float32)
    return x, (2 * np.arange(n + 1)).astype(np.uint32), np.sort(adj, 1).ravel(), (v // 3).astype(np.uint32)


def test_not_in_the_calls_pool():
    import torch
    watch = _PoolWatch()
    torch.cuda.synchronize()
    used = watch.reset()
    ests = [A.Estimator(44, seed) for seed in range(3)]
    for graphs in (10, 3000, 200):  # workspaces grow and are reused
        x, off, adj, gid = _batch(graphs)
        for e in ests:
            e.predict(x, off, adj, gid, graphs)
            e.train_step(x, off, adj, gid, np.ones(graphs, np.float32), lr=1e-3)
    assert watch.high() == used


def test_memory_comes_back():
    import torch
    x, off, adj, gid = _batch(100_000)  # over 1 GB of workspace

    def free():
        gc.collect()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    e = A.Estimator(44, 0)
    before = free()
    y = e.predict(x, off, adj, gid, 100_000)
    assert before - free() > 1 << 30
    del e
    assert before - free() < 300 << 20  # what the pool keeps for the next estimator
    e = A.Estimator(44, 0)
    assert np.array_equal(e.predict(x, off, adj, gid, 100_000), y)
