"""GPU tests of runs for which a faster route's buffers do not fit: they take
the route that needs less, with the same results.  Device memory is limited on
the host: while a run is on, the library's allocations (cudaMallocAsync) come
from a pool of a fixed size, which refuses what does not fit."""
import contextlib

import numpy as np
import pytest

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def device_memory(mb, device=0):
    """Limits the library's device memory to mb MiB (a multiple of 32: a pool grows in such steps)."""
    from cuda.bindings import runtime as rt

    def call(f, *args):
        err, *out = f(*args)
        assert err == rt.cudaError_t.cudaSuccess, err
        return out[0] if out else None
    props = rt.cudaMemPoolProps()
    props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
    props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
    props.location.id = device
    props.maxSize = mb * MB
    before = call(rt.cudaDeviceGetMemPool, device)
    pool = call(rt.cudaMemPoolCreate, props)
    call(rt.cudaDeviceSetMemPool, device, pool)
    try:
        yield
    finally:
        call(rt.cudaDeviceSetMemPool, device, before)
        call(rt.cudaDeviceSynchronize)
        call(rt.cudaMemPoolDestroy, pool)


@pytest.fixture(scope="module")
def far():
    """A dense graph of four labels among 4,000,000 vertices, so that local-count matrices are large beside the rest,
    and a tree whose ends have one label: a triangle is its quotient."""
    rng = np.random.default_rng(2)
    e = np.unique(np.sort(np.minimum(rng.integers(0, 2500, (250_000, 2)), rng.integers(0, 2500, (250_000, 2))), 1), axis=0)
    labels = np.full(4_000_000, 9)
    labels[:2500] = rng.integers(0, 4, 2500)
    dg = A.DeviceGraph(A.HostGraph.from_edges(len(labels), labels, e[e[:, 0] != e[:, 1]]))
    q = A.HostGraph.from_edges(5, [0, 1, 2, 0, 3], [[0, 1], [1, 2], [2, 3], [3, 4]])
    with contextlib.closing(dg), contextlib.closing(A.CandidateSpace(dg, q)) as cs:
        whole = A.adaptive_share_join(cs, mode=A.MODE_LOCAL, time_limit_s=300.0)  # a run with a limit enumerates the tree
        assert whole.count > 2 ** 29
        yield dg, q, cs, whole


def test_quotients_do_not_fit(far):
    dg, q, cs, whole = far
    with device_memory(256):  # the query's matrix has 160 MB, the quotient's 128 MB
        r = A.adaptive_share_join(cs, mode=A.MODE_LOCAL)
    assert r.intersections == 0  # the tree was enumerated: a tree's levels have one list each
    assert r.count == whole.count and np.array_equal(r.local_counts, whole.local_counts)
    r = A.adaptive_share_join(cs, mode=A.MODE_LOCAL)
    assert r.intersections > 0  # its quotient, a triangle with a leaf, was
    assert r.count == whole.count and np.array_equal(r.local_counts, whole.local_counts)


def test_quotients_of_a_batch_do_not_fit(far):
    dg, q, cs, whole = far
    edge = A.HostGraph.from_edges(2, [0, 1], [[0, 1]])
    want = A.match(dg, edge, A.MODE_LOCAL)
    with device_memory(320):  # both matrices have 224 MB
        counts, status, local = A.run_batch_local(dg, [edge, q])
    assert status.tolist() == [A.OK, A.OK] and counts.tolist() == [want.count, whole.count]
    assert np.array_equal(local[0], want.local_counts) and np.array_equal(local[1], whole.local_counts)

@pytest.fixture(scope="module")
def star():
    """A centre with four leaves of one label: 15 terms, each with weights, list sums and ways up."""
    rng = np.random.default_rng(3)
    n = 400_000
    e = np.unique(np.sort(rng.integers(0, n, (2_000_000, 2)), 1), axis=0)
    dg = A.DeviceGraph(A.HostGraph.from_edges(n, rng.integers(0, 2, n), e[e[:, 0] != e[:, 1]]))
    q = A.HostGraph.from_edges(5, [0, 1, 1, 1, 1], [[0, i] for i in range(1, 5)])
    with contextlib.closing(dg), contextlib.closing(A.CandidateSpace(dg, q)) as cs:
        yield dg, q, cs, A.adaptive_share_join(cs, mode=A.MODE_LOCAL)


@pytest.mark.parametrize("mb", [64, 128])
def test_tree_program_does_not_fit(star, mb):
    dg, q, cs, whole = star
    with device_memory(mb):
        r = A.adaptive_share_join(cs, mode=A.MODE_LOCAL)
    assert whole.list_bytes == 0 and r.list_bytes > 0  # enumerated
    assert r.count == whole.count and np.array_equal(r.local_counts, whole.local_counts)


def test_tree_program_of_a_batch_does_not_fit(star):
    dg, q, cs, whole = star
    edge = A.HostGraph.from_edges(2, [0, 1], [[0, 1]])
    want = A.match(dg, edge, A.MODE_LOCAL)
    with device_memory(192):
        counts, status, local = A.run_batch_local(dg, [q, edge])
    assert status.tolist() == [A.OK, A.OK] and counts.tolist() == [whole.count, want.count]
    assert np.array_equal(local[0], whole.local_counts) and np.array_equal(local[1], want.local_counts)


def test_gathered_entries_do_not_fit():
    k = 500_000  # disjoint cycles of six labels: a matrix of 144 MB, 36 MB of gathered entries
    base = 6 * np.arange(k)[:, None]
    edges = np.concatenate([base + [[i, (i + 1) % 6]] for i in range(6)])
    dg = A.DeviceGraph(A.HostGraph.from_edges(6 * k, np.tile(np.arange(6), k), edges))
    q = A.HostGraph.from_edges(6, range(6), [[i, (i + 1) % 6] for i in range(6)])
    want = np.zeros((6 * k, 6), np.uint64)
    want[np.arange(6 * k), np.tile(np.arange(6), k)] = 1
    with contextlib.closing(dg), contextlib.closing(A.CandidateSpace(dg, q)) as cs:
        for mb in (160, 512):
            with device_memory(mb):
                r = A.adaptive_share_join(cs, mode=A.MODE_LOCAL)
            assert r.count == k and np.array_equal(r.local_counts, want)


# four million rows: keys 32 MB, the sort's two key buffers 64 MB and its output 48 MB
@pytest.mark.parametrize("mb", [256, 128, 96, 64])
def test_sort_does_not_fit(mb):
    a, c = np.arange(2000), np.arange(2001, 4001)
    edges = np.stack([np.concatenate([a, c]), np.full(4000, 2000)], 1)
    dg = A.DeviceGraph(A.HostGraph.from_edges(4001, [0] * 2000 + [1] + [2] * 2000, edges))
    q = A.HostGraph.from_edges(3, [0, 1, 2], [[0, 1], [1, 2]])
    with contextlib.closing(dg), contextlib.closing(A.CandidateSpace(dg, q)) as cs:
        with device_memory(mb):
            rows = A.adaptive_share_join(cs, mode=A.MODE_EMBED, emb_capacity=4_000_000).embeddings
    assert np.array_equal(rows, np.stack([np.repeat(a, 2000), np.full(4_000_000, 2000), np.tile(c, 2000)], 1))
