"""GPU tests of the stream that set intersections run on: they neither wait for
nor hold up the work that a program has on the legacy default stream (PyTorch's
default), and calls from several threads, which have a stream each, run side by
side."""
import concurrent.futures as cf

import numpy as np
import pytest
import torch

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu


def _sets(seed):
    rng = np.random.default_rng(seed)
    sets = [[np.unique(rng.integers(0, 4000, 1000, dtype=np.uint32)) for _ in range(3)] for _ in range(8)]
    return sets, [np.intersect1d(np.intersect1d(a, b), c) for a, b, c in sets]


def test_beside_the_default_stream():
    sets, want = _sets(5)
    A.leapfrog_join(sets)
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000_000)  # a spin of about half a second on the default stream
    done = torch.cuda.Event()
    done.record()
    got = A.leapfrog_join(sets)
    assert not done.query()
    torch.cuda.synchronize()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_threads():
    cases = [_sets(seed) for seed in range(12)]
    for _ in range(3):  # threads come and go
        with cf.ThreadPoolExecutor(4) as ex:
            for got, (_, want) in zip(ex.map(lambda c: A.leapfrog_join(c[0]), cases), cases):
                assert all(np.array_equal(a, b) for a, b in zip(got, want))
