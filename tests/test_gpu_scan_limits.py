"""Limits of the exact scan (needs a B200): rows too wide for the interface are
refused whatever the batch, so that support does not depend on the data."""
import numpy as np
import pytest

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import _capi, pickling

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,fits", [(2800, True), (3072, False)])
def test_row_width(tmp_path, dim, fits):
    rng = np.random.default_rng(dim)
    n = 5000
    x = rng.standard_normal((n, dim)).astype(np.float32)
    (tmp_path / "bf.bin").write_bytes(pickling.bf_rows_to_file(x, np.arange(n, dtype=np.uint64), n, dim))
    g = H.BFIndex("l2", dim)
    g.load_index(str(tmp_path / "bf.bin"))
    for nq in (1, 7, 100):  # the last batch is large enough for the tensor-core route
        q = x[:nq] + np.float32(0.01)
        if fits:
            assert np.array_equal(g.knn_query(q, 5)[0][:, 0], np.arange(nq))
        else:
            with pytest.raises(_capi.HnswGpuError, match="invalid configuration"):
                g.knn_query(q, 5)
