"""The certified exact scan on rows that bf16 holds exactly, where only the
tensor cores' accumulation stands between the scores and the proof (needs a
B200): byte-valued rows with near duplicates, and products that all lie just
under the last bit kept of the first.  Bit-identical to BruteforceSearch."""
import numpy as np
import pytest

from test_gpu_bf_forms import _pair, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("dim", [100, 768])
def test_bytes_with_near_duplicates(tmp_path, space, dim):
    rng = np.random.default_rng(dim)
    n = 8000
    base = rng.integers(0, 255, (n // 40, dim))
    x = base[rng.integers(0, len(base), n)] + (rng.random((n, dim)) < rng.choice([0.002, 0.02, 0.2], (n, 1)))
    q = x[rng.integers(0, n, 1000)] + (rng.random((1000, dim)) < 0.01)
    g, o = _pair(tmp_path, x.astype(np.float32), space)
    for k in (1, 10, 100):
        _same(g, o, np.minimum(q, 255).astype(np.float32), k)


@pytest.mark.parametrize("space", ["l2", "ip"])
def test_products_under_the_last_bit(tmp_path, space):
    rng = np.random.default_rng(5)
    n, dim, near = 8000, 768, 150
    x = rng.choice([-0.5, 0.25, 0.5], (n, 1)) * np.eye(1, dim) + 2.0 ** -6 * rng.integers(-1, 2, (n, dim))
    rows = rng.permutation(n)[:near]  # 1 and up to 767 products of 0.996 * 2^-23
    x[rows] = np.where(rng.random((near, dim)) < rng.random((near, 1)), 1.9921875 * 2.0 ** -13, 0)
    x[rows, 0] = 1
    q = np.full((200, dim), 2.0 ** -11)
    q[:, 0] = 1
    q[1:, 1:] *= rng.random((199, dim - 1)) < 0.9
    g, o = _pair(tmp_path, x.astype(np.float32), space)
    for k in (1, 10, 40):
        _same(g, o, q.astype(np.float32), k)
