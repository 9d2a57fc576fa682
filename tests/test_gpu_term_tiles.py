"""Training kernels at the edges of their tiles (needs a B200): gradients of
any sample count against the float64 oracle, to 1e-4 of the largest entry (the
bound of the existing gradient test), and training over ragged last batches."""
import numpy as np
import pytest

from hnsw_rabitq_b200 import learned
from oracle import term_mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 1000])
def test_gradient_tiles(n):
    rng = np.random.default_rng(n)
    f = rng.normal(size=(n, learned.F)).astype(np.float32)
    y = (rng.random(n) < 0.5).astype(np.float32)
    p = learned.init_params(rng.normal(size=(64, learned.F)), n)
    loss, g = learned.loss_grad(p, f, y, pos_weight=1.5)
    ol, og = term_mlp.loss_grad(p, f, y, 1.5)
    assert abs(loss - ol) <= 1e-5 * max(1.0, abs(ol))
    assert np.max(np.abs(g - og)) <= 1e-4 * np.max(np.abs(og))


@pytest.mark.parametrize("n,batch", [(300, 256), (1000, 100), (129, 1024)])
def test_training_is_deterministic(n, batch):
    rng = np.random.default_rng(n)
    f = rng.normal(size=(n, learned.F)).astype(np.float32)
    y = (f[:, 0] > 0).astype(np.float32)
    a = learned.train(f, y, epochs=5, batch=batch, seed=3)
    b = learned.train(f, y, epochs=5, batch=batch, seed=3)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert a[1][-1] < a[1][0]
