"""GPU test of the estimator's training step at node counts where the weight
gradients' product changes form: one chunk of nodes, the first split, ragged
last chunks, more chunks than splits.

The network is set up so that every stored value is exact: identity weights,
zero biases, small whole features.  The gradients are then sums, of one sign, of
products of bf16 values known beforehand.  A first step with learning rate 0
only fills Adam's moments with the batch's gradient g1; a second step on a small
batch (gradient g2) with learning rate 1 moves the weights by a function of
g1 / g2.  Tolerance: fp32 sums of up to 12,000 terms of one sign err by at most
12,000 x 2^-24 < 10^-3 of the sum, and the function's slope is below 1."""
import numpy as np
import pytest

import asdmatch_b200 as A

pytestmark = pytest.mark.gpu

H, F = 128, 20
WO = np.where(np.arange(H) % 2 == 0, 1.0, -2.0).astype(np.float32)


def _batch(nodes, seed):
    """Paths of three nodes (the last graph takes what is left): inputs and the exact weight gradients per layer."""
    rng = np.random.default_rng(seed)
    ng = max(1, nodes // 3)
    gid = np.minimum(np.arange(nodes) // 3, ng - 1)
    src = np.nonzero(gid[:-1] == gid[1:])[0]
    both = np.concatenate([np.stack([src, src + 1], 1), np.stack([src + 1, src], 1)])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    off = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=nodes))]).astype(np.uint32)
    x = rng.integers(0, 4, (nodes, F)).astype(np.float32)
    h = np.zeros((nodes, H))
    h[:, :F] = x
    around = np.zeros_like(h)
    np.add.at(around, both[:, 0], h[both[:, 1]])
    pooled = np.zeros((ng, H))
    np.add.at(pooled, gid, h)
    r = rng.integers(1, 3, ng).astype(np.float32)
    target = (pooled @ WO - r).astype(np.float32)
    dy = (np.float32(2) * r / np.float32(ng)).astype(np.float32)
    dz = A.from_bf16_bits(A.to_bf16_bits(dy[gid][:, None] * WO)).reshape(nodes, H).astype(np.float64) * (h > 0)
    grad = dz.T @ np.concatenate([h, around], 1)  # every layer's: its input and its mask are the features
    return (x, off, both[:, 1].astype(np.uint32), gid.astype(np.uint32), target), grad


@pytest.mark.parametrize("nodes", [1, 63, 64, 65, 128, 129, 192, 255, 1000, 8191, 8192, 8193, 8257, 12_000])
def test_weight_gradients(nodes):
    est = A.Estimator(F)
    p = np.zeros(3 * 2 * H * H + 4 * H + 1, np.float32)
    for k in range(3):
        p[k * 2 * H * H:(k + 1) * 2 * H * H] = np.concatenate([np.eye(H), np.zeros((H, H))], 1).ravel()
    p[3 * 2 * H * H + 3 * H:-1] = WO
    est.set_params(p)
    b1, g1 = _batch(nodes, nodes)
    b2, g2 = _batch(9, nodes + 1)
    est.train_step(*b1, lr=0.0)
    assert np.array_equal(est.params(), p)
    est.train_step(*b2, lr=1.0)
    m = (0.09 * g1 + 0.1 * g2) / (1 - 0.81)
    v = (0.000999 * g1 * g1 + 0.001 * g2 * g2) / (1 - 0.998001)
    want = m / (np.sqrt(v) + 1e-8)
    for k in range(3):
        moved = (p - est.params())[k * 2 * H * H:(k + 1) * 2 * H * H].reshape(H, 2 * H)
        assert np.max(np.abs(moved - want)) <= 1e-3, k
