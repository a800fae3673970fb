"""GPU test of the batched intersection at the edges of a driver chunk (32 to
1,024 elements) and of the warp-wide cursor search: problems of very different
sizes in one call, empty lists, one list, 32 lists; against numpy."""
import numpy as np
import pytest

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu


def _check(sets):
    got = A.leapfrog_join(sets)
    for lists, g in zip(sets, got):
        want = np.zeros(0, np.uint32)
        if lists:
            want = np.asarray(lists[0], np.uint32)
            for l in lists[1:]:
                want = np.intersect1d(want, l, assume_unique=True)
        assert np.array_equal(g, want)


@pytest.mark.parametrize("driver", [1, 31, 32, 33, 63, 64, 65, 1023, 1024, 1025, 70_000])
@pytest.mark.parametrize("ratio", [1, 8, 9, 400])
def test_one_problem(driver, ratio):
    rng = np.random.default_rng(driver * 1000 + ratio)
    other = min(driver * ratio, 4_000_000)
    top = 3 * other + 7
    lists = [np.unique(rng.integers(0, top, driver, dtype=np.uint32)),
             np.unique(rng.integers(0, top, other, dtype=np.uint32)),
             np.arange(0, top, 2, dtype=np.uint32)]
    _check([lists, lists[::-1], lists[:1]])


def test_mixed_problems():
    rng = np.random.default_rng(5)
    sets = [[], [np.zeros(0, np.uint32), np.arange(9, dtype=np.uint32)], [np.array([0xFFFFFFFE, 0xFFFFFFFF], np.uint32)] * 3]
    for k in (1, 2, 5, 32):
        for n in (1, 40, 3000):
            sets.append([np.unique(rng.integers(0, 2 * n + 3, n, dtype=np.uint32)) for _ in range(k)])
    # disjoint, identical, and interleaved blocks
    a = np.arange(100_000, dtype=np.uint32)
    sets += [[a, a + 100_000], [a, a], [a[a % 64 < 32], a[a % 64 >= 32]], [a, a[::997]], [a[50_000:], a[:50_001]]]
    _check(sets)
    _check(sets * 40)  # longer chunks
