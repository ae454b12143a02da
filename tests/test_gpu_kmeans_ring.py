"""The tensor-core k-means where its centroids leave room for a row ring of two, three
and more stages: many clusters of many coordinates, with one tile and many, one and
two accumulators, a last coordinate group that is whole and one that is not.  Hashes of
landmarks and initial labels and the label matrix equal the CPU restatement's."""

import numpy as np
import pytest

from kodama_gb300 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [
    (271, 141, 300), (225, 133, 300), (220, 148, 520), (595, 102, 300), (849, 105, 300), (2373, 96, 300), (1200, 87, 300),
    (900, 130, 200), (400, 256, 128), (600, 200, 160), (531, 65, 300), (700, 64, 512), (900, 80, 400), (1500, 112, 256),
    (700, 250, 100), (5000, 90, 300)])
@pytest.mark.parametrize("runs", [1, 5])
def test_few_stages_match_oracle(kg, orc, n, d, k, runs):
    x, _ = datasets.gaussian_mixture(n=n, d=d, seed=n + k)
    rng = np.random.default_rng(n)
    gi = np.stack([(np.arange(n) + s) % n for s in (1, 2, 3, 5, 8)], axis=1).astype(np.int32)
    gd = np.sort(rng.random((n, 5), dtype=np.float32), axis=1)
    kw = dict(runs=runs, cycles=1, landmarks=10000, splitting=k, graph_neighbors=5, folds=3, knn_k=3, seed=11)
    r = orc.kodama_matrix_graph_data(x, gi, gd, 0, threads=8, **kw)
    for _ in range(2):
        g = kg.KODAMA_matrix(x, graph=(gi, gd), index_base=0, **kw)
        assert np.array_equal(g.run_hashes, r.hashes)
        assert np.array_equal(g.res, r.res)
