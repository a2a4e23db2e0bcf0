"""Minibatch training of the controller network (one cluster per epoch, or one launch per batch) against
FP64 Adam on the FP64 gradient of oracle/mlp.py, over batch sizes that leave CTAs without samples, end in
a batch of one, or take several chunks per CTA.

Tolerance: the FP32 gradient is within 1e-6 of the FP64 one (1e-5 in its own check) and a weight moves by
at most lr per step; a weight whose gradient is rounding noise may move the other way, so the bound is
1e-4 of the weights' norm."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def _orders(n, epochs, seed):
    mask, s, p = (1 << 64) - 1, seed, list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            p[i], p[j] = p[j], p[i]
        yield np.array(p)


@pytest.mark.parametrize("n,batch,epochs", [(300, 300, 1), (1000, 256, 2), (257, 256, 2), (37, 5, 3), (9, 1, 1), (5000, 2560, 2),
                                            (5000, 2561, 2)])
def test_training_follows_fp64_adam(gpu_lib, n, batch, epochs):
    from mpc_gb300.capi import MLP
    rng = np.random.default_rng(n + batch)
    w = (rng.standard_normal(omlp.NW) * 0.2).astype(np.float32)
    X = rng.standard_normal((n, 16)).astype(np.float32) * 3 + 1
    y = (np.sin(X[:, 0]) + 0.3 * X[:, 1] * X[:, 2] / 9).astype(np.float32)
    norm = np.concatenate([np.full(16, 1.0), np.full(16, 3.0), [0.1, 0.7]]).astype(np.float32)
    mlp = MLP(0)
    mlp.set_normalization(norm[:16], norm[16:32], norm[32], norm[33])
    mlp.weights = w
    loss = mlp.train(X, y, epochs=epochs, batch=batch, lr=1e-3, seed=5)
    got = mlp.weights
    mlp.close()
    ref, m, v, t, total = w.astype(np.float64), 0.0, 0.0, 0, 0.0
    b1, b2, lr, eps = (float(np.float32(k)) for k in (0.9, 0.999, 1e-3, 1e-8))
    for order in _orders(n, epochs, 5):
        total = 0.0
        for k in range(0, n, batch):
            at = order[k:k + batch]
            l, g = omlp.loss_grad(ref, X[at], y[at], norm)
            total += l * len(at) / n
            t += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            ref = ref - lr * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + eps)
    assert abs(loss / total - 1) < 1e-4
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-4
