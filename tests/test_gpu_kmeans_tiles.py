"""The tensor-core k-means (kmeans.cu) where its splits can go wrong: row counts
around the 128-row tiles, cluster counts around the 16 / 32 / 64 / 256 / 512
column splits, coordinate counts around the 64-coordinate stages, rows with
many candidates (far from the origin, ties), values outside the range of the
error bound, and a batch whose assignments do not fit in shared memory.  The
landmark k-means of KODAMA.matrix is compared through the hashes of landmarks
and initial labels, with the whole result, against the CPU restatement: equal
bit for bit, so the tolerance is 0."""
import numpy as np
import pytest

from kodama_gb300 import datasets

pytestmark = pytest.mark.gpu


def _check(kg, orc, x, splitting, landmarks=10000, runs=2):
    n = x.shape[0]
    rng = np.random.default_rng(n)
    # any graph will do: the k-means reads the data alone
    gi = np.stack([(np.arange(n) + s) % n for s in (1, 2, 3, 5, 8)], axis=1).astype(np.int32)
    gd = np.sort(rng.random((n, 5), dtype=np.float32), axis=1)
    kw = dict(runs=runs, cycles=1, landmarks=landmarks, splitting=splitting, graph_neighbors=5, folds=3, knn_k=3,
              seed=11)
    g = kg.KODAMA_matrix(x, graph=(gi, gd), index_base=0, **kw)
    r = orc.kodama_matrix_graph_data(x, gi, gd, 0, threads=8, **kw)
    assert np.array_equal(g.run_hashes, r.hashes)
    assert np.array_equal(g.res, r.res)


@pytest.mark.parametrize("n,d,k", [(170, 1, 2), (171, 15, 16), (172, 16, 17), (340, 17, 33), (600, 63, 64),
                                   (600, 64, 65), (700, 65, 128), (700, 129, 31), (900, 256, 48), (1100, 9, 256),
                                   (1100, 9, 257), (1500, 24, 511), (1500, 24, 512), (1200, 6, 600),
                                   (500, 300, 20)])
def test_kmeans_edges(kg, orc, n, d, k):
    x, _ = datasets.gaussian_mixture(n=n, d=d, seed=n + k)
    _check(kg, orc, x, k)


@pytest.mark.parametrize("kind", ["far", "ties", "huge", "infinite"])
@pytest.mark.parametrize("k", [20, 100])
def test_kmeans_hard_values(kg, orc, kind, k):
    x, _ = datasets.gaussian_mixture(n=900, d=12, seed=k)
    if kind == "far":
        x = x + np.float32(3000.0)
    elif kind == "ties":
        x = np.round(x / 4).astype(np.float32)
        x[300:600] = x[:300]
    elif kind == "huge":
        x = x * np.float32(1e18)
    else:
        x[::50, 3] = np.inf
    _check(kg, orc, np.ascontiguousarray(x, np.float32), k)


def test_kmeans_many_rows(kg, orc):
    # 58000 rows per problem, 300 clusters: one pass per launch
    x, _ = datasets.gaussian_mixture(n=60000, d=40, clusters=25, seed=6)
    _check(kg, orc, x, 300, landmarks=58000)
