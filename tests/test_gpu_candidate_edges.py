"""GPU tests of the candidate-edge lists (K3): the chunked fill against the
exact two-scan form, by the device's digest, on graphs whose label runs are
much longer than a chunk, all of one entry, or mixed; and against lists written
down with numpy at sizes around the chunk length."""
import numpy as np
import pytest

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu


def _hubs(hubs, leaves):
    """Every hub (label 0) is adjacent to every leaf (label 1)."""
    labels = np.array([0] * hubs + [1] * leaves)
    edges = np.stack(np.meshgrid(np.arange(hubs), hubs + np.arange(leaves), indexing="ij"), -1).reshape(-1, 2)
    return A.HostGraph.from_edges(hubs + leaves, labels, edges), edges


@pytest.mark.parametrize("make", [
    lambda: (_hubs(3, 400_000)[0], [0, 1, 1], [[0, 1], [0, 2]]),
    lambda: (_hubs(900, 1300)[0], [0, 1, 0], [[0, 1], [1, 2]]),
    lambda: (A.HostGraph.chung_lu(300_000, 1_500_000, 2.1, 3, 1.0, 5), None, 6),
    lambda: (A.HostGraph.chung_lu(300_000, 1_500_000, 2.9, 40, 0.2, 6), None, 12),
])
def test_chunked_fill_equals_two_scans(make):
    g, labels, shape = make()
    dg = A.DeviceGraph(g)
    tune = dg.tuning()
    qs = [A.HostGraph.from_edges(len(labels), labels, shape)] if labels else \
        [g.random_walk_query(shape, 17 + i) for i in range(12)]
    digests = []
    for cap in (tune["padded_cap_log2"], 20):
        dg.set_tuning(tune["enum_min_blocks"], tune["lane_leaf_max"], padded_cap_log2=cap)
        css = A.candidate_spaces(dg, qs) + [A.CandidateSpace(dg, q) for q in qs]
        digests.append([cs.digest()[0] for cs in css])
        if cap != 20:
            assert not any(cs.digest()[1] & A.CS_TWO_SCAN for cs in css)
        elif shape != 12:  # (the graph of 40 labels stays below 2^20 entries: it compares group and single builds)
            assert any(cs.digest()[1] & A.CS_TWO_SCAN for cs in css)
        for cs in css:
            cs.close()
    dg.close()
    assert digests[0] == digests[1]
    assert digests[0][:len(qs)] == digests[0][len(qs):]


# entries per direction around the chunk's length (128 for small groups) and multiples of it
@pytest.mark.parametrize("hubs,leaves", [(1, 1), (1, 127), (1, 128), (1, 129), (2, 64), (3, 43), (4, 160), (127, 2),
                                         (128, 1), (33, 65), (1, 4097)])
def test_lists_of_a_biclique(hubs, leaves):
    g, edges = _hubs(hubs, leaves)
    dg = A.DeviceGraph(g)
    cs = A.CandidateSpace(dg, A.HostGraph.from_edges(2, [0, 1], [[0, 1]]))
    off, ids = cs.candidate_edge(0, 1)
    assert np.array_equal(off, np.arange(hubs + 1) * leaves)
    assert np.array_equal(ids, edges[:, 1])
    off, ids = cs.candidate_edge(1, 0)
    assert np.array_equal(off, np.arange(leaves + 1) * hubs)
    assert np.array_equal(ids, np.tile(np.arange(hubs), leaves))
    cs.close()
    dg.close()


# around the 2^20 possible entries beyond which the short form reads its length back, and the 2^16 items
# (both directions' candidates and an end each) and 2^22 possible entries beyond which the chunked form runs
@pytest.mark.parametrize("hubs,leaves", [(512, 1023), (512, 1024), (512, 1025), (2, 65_531), (2, 65_532), (2, 65_533),
                                         (1447, 1449), (1448, 1449)])
def test_short_form_limits(hubs, leaves):
    test_lists_of_a_biclique(hubs, leaves)
