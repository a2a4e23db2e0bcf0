"""A batch larger than the set is the whole set, up to the largest int."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_beyond_the_set(gpu_lib):
    from mpc_gb300.capi import MLP
    rng = np.random.default_rng(3)
    X, y = rng.standard_normal((3000, 16)).astype(np.float32), rng.standard_normal(3000).astype(np.float32)
    out = []
    for batch in (3000, 100000, 2 ** 31 - 1):
        net = MLP(seed=5)
        loss = net.train(X, y, epochs=2, batch=batch)
        out.append((loss, net.weights))
        net.close()
    for loss, w in out[1:]:   # gradients are added by atomics: FP32 rounding
        assert loss == pytest.approx(out[0][0], rel=1e-5) and np.allclose(w, out[0][1], atol=1e-5)
    assert out[0][0] > 0
