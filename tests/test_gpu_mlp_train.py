"""Training the picker's network against a float64 restatement of its steps,
at the sizes where the cluster kernel's tiles meet (8 rows of a CTA, 128 of a
tile, several tiles to a batch) and beyond the largest batch it takes."""
import numpy as np
import pytest

from nvshmem_b200 import picker as P
from oracle import mlp_ref as R

pytestmark = pytest.mark.gpu

MASK64 = (1 << 64) - 1


def mix64(x):
    x = (x + 0x9E3779B97F4A7C15) & MASK64
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & MASK64
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & MASK64
    return x ^ (x >> 31)


def train64(p, X, Y, M, epochs, batch, lr, seed, mean, std):
    n, m, v, step, curve = len(X), np.zeros_like(p), np.zeros_like(p), 0, []
    for e in range(epochs):
        perm, st = list(range(n)), (seed * 0x100000001B3 + e) & MASK64
        for i in range(n - 1, 0, -1):
            j = mix64(st) % (i + 1)
            st += 1
            perm[i], perm[j] = perm[j], perm[i]
        total, nb = 0.0, 0
        for b in range(0, n, batch):
            rows = perm[b:b + batch]
            nb += 1
            if M[rows].sum() <= 0:
                continue
            loss, g = R.loss_grad(p, X[rows], Y[rows], M[rows], mean, std)
            total += loss
            step += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            p = p - lr * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        curve.append(total / nb)
    return p, np.array(curve)


@pytest.mark.parametrize("n,batch", [(1, 1), (7, 8), (130, 17), (257, 128), (700, 300), (600, 512), (1300, 600)])
def test_training_steps_match_float64(n, batch):
    rng = np.random.default_rng(n)
    X = (rng.normal(size=(n, 6)) * 3 + 5).astype(np.float32)
    Y = rng.normal(size=(n, 12)).astype(np.float32)
    M = (rng.random((n, 12)) > 0.15).astype(np.float32)
    M[n // 2] = 0.0  # a row without any measured variant (with one row: no step at all)
    mean, std = X.mean(0), np.maximum(X.std(0), 1e-3)
    nets = [P.MLP(seed=3) for _ in range(3)]  # the third lies outside the library's own array
    got = []
    for net in nets:
        net.set_normalization(mean, std)
        p0 = net.params()
        curve = net.train(X, Y, M, epochs=3, batch=batch, lr=2e-3, seed=9)
        got.append((net.params(), curve))
    want, wcurve = train64(p0.astype(np.float64), X, Y, M, 3, batch, 2e-3, 9, mean.astype(np.float64),
                           std.astype(np.float64))
    for p, curve in got:
        # float32 rounding of a few dozen Adam steps (the bias corrections
        # alone carry 1e-5), and a ReLU that falls on the other side
        assert np.linalg.norm(p - want) <= 5e-4 * np.linalg.norm(want)
        assert np.allclose(curve, wcurve, rtol=1e-3, atol=1e-6)
    if batch <= 512:  # one cluster sums in a fixed order
        assert all(np.array_equal(p, got[0][0]) for p, _ in got)
    for net in nets:
        net.close()


def test_a_table_larger_than_the_kept_memory():
    rng = np.random.default_rng(5)
    n = 200_000  # 4.8 MB of features, 9.6 MB of outputs: more than a network keeps
    X = rng.normal(size=(n, 6)).astype(np.float32)
    net = P.MLP(seed=4)
    small = net.forward(X[-40:])
    assert np.array_equal(net.forward(X)[-40:], small)
    net.close()
