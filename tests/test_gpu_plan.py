"""Landmark planning at its limits: few and many strata (their state in shared or
global memory), more initial centroids than an engine block holds outputs, as many
as there are landmarks, and sizes around the 32-step batches of the sampling.  The
runs' landmark, start and fold hashes and results are the CPU restatement's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,landmarks,splitting,runs", [
    (37, 20, 2, 3), (60, 40, 50, 3), (64, 63, 3, 2), (65, 40, 1, 2), (1000, 750, 100, 3), (3000, 2500, 700, 2),
    (2600, 2500, 2100, 1), (5003, 1200, 7, 2),
])
def test_planned_runs_match_oracle(kg, orc, n, landmarks, splitting, runs):
    rng = np.random.default_rng(n + splitting)
    x = rng.standard_normal((n, 4)).astype(np.float32)
    K = min(10, n - 1)
    gi, gd = orc.exact_knn(x, K, threads=8)
    kw = dict(runs=runs, cycles=2, landmarks=landmarks, splitting=splitting, graph_neighbors=K, folds=3, knn_k=5)
    a = orc.kodama_matrix_graph_data(x, gi, gd, 0, seed=7, threads=4, materialize=1, **kw)
    b = kg.KODAMA_matrix(x, graph=(gi, gd), index_base=0, seed=7, materialize_graph=True, **kw)
    assert np.array_equal(a.hashes, b.run_hashes)
    for f in ("res", "acc", "v", "run_counters", "cycle_diag"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
