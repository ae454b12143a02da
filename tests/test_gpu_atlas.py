"""The atlas k-means' update step at its limits: clusters larger than the list of
members held at a time, one column to more than a thread takes, warps without rows,
empty clusters.  The atlas labels decide every run's landmarks, so the run hashes
and results equal the CPU restatement's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,splitting", [(40, 1, 5), (513, 3, 7), (20011, 2, 2), (1000, 513, 6), (700, 1024, 3)])
def test_atlas_matches_oracle(kg, orc, n, d, splitting):
    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d)).astype(np.float32)
    x[: n // 2] = x[0]  # half the rows alike: one large cluster, others empty
    K = min(8, n - 1)
    g = np.argsort(rng.random((n, 2 * K)), axis=1)[:, :K]  # any graph: distinct neighbours near the row
    gi = ((np.arange(n)[:, None] + 1 + g) % n).astype(np.int32)
    gd = np.sort(rng.random((n, K)).astype(np.float32), axis=1)
    kw = dict(runs=2, cycles=2, landmarks=max(20, min(n // 2, 3000)), splitting=splitting, graph_neighbors=K, folds=3,
              knn_k=4)
    a = orc.kodama_matrix_graph_data(x, gi, gd, 0, seed=9, threads=8, materialize=1, **kw)
    b = kg.KODAMA_matrix(x, graph=(gi, gd), index_base=0, seed=9, materialize_graph=True, **kw)
    assert np.array_equal(a.hashes, b.run_hashes)
    for f in ("res", "acc", "v", "run_counters", "cycle_diag"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
