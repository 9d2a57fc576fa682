"""Scans of four indexes from four threads, whose selection kernels take shared
memory of different sizes (needs a B200): every call succeeds and returns what
it returns alone."""
import threading

import numpy as np
import pytest

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import pickling

pytestmark = pytest.mark.gpu


def _index(path, n, dim, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    path.write_bytes(pickling.bf_rows_to_file(x, np.arange(n, dtype=np.uint64), n, dim))
    g = H.BFIndex("l2", dim)
    g.load_index(str(path))
    return g, rng.standard_normal((128, dim)).astype(np.float32)


@pytest.mark.parametrize("prec", ["fp32", "bf16"])
def test_indexes_of_four_threads(tmp_path, prec):
    jobs = [(*_index(tmp_path / f"{i}.bin", 5000, 1024, i), k) for i, k in enumerate((5, 200, 20, 150))]
    want, errors = [], []
    for g, q, k in jobs:
        g.precision = prec
        want.append(g.knn_query(q, k))

    def loop(i):
        g, q, k = jobs[i]
        try:
            for _ in range(1500):
                l, d = g.knn_query(q, k)
                assert np.array_equal(l, want[i][0]) and np.array_equal(d, want[i][1])
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
