"""The tensor-core neighbour search (knn_tc.cu) where its splits can go wrong:
row counts around the 128-query and 256-candidate tiles, list capacities
(128 / 256 / 512 entries), coordinate counts around the 16-wide steps, inner
products, candidates of other folds, rows that are no 16-byte vectors, and
values outside the range its error bound holds for.  Everything equals the CPU
restatement bit for bit (the search is certified per row), so the tolerance
is 0."""
import numpy as np
import pytest

from kodama_gb300 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,K,metric", [
    (256, 1, 35, 2), (257, 8, 36, 2), (385, 256, 111, 2), (512, 17, 112, 2), (513, 33, 222, 2), (640, 31, 223, 2),
    (255, 5, 30, 2), (1025, 130, 100, 2), (256, 7, 20, 1), (700, 48, 100, 1), (511, 19, 35, 0), (1300, 257, 30, 0),
    (2049, 100, 112, 0)])
def test_graph_edges(kg, orc, n, d, K, metric):
    x, _ = datasets.gaussian_mixture(n=n, d=d, seed=n + K)
    gi, gd = kg.knn_graph(x, K, metric=metric)
    ri, rd = orc.exact_knn(x, K, threads=8) if metric == 2 else orc.exact_knn_metric(x, K, metric, threads=8)
    assert np.array_equal(gi, ri)
    assert np.array_equal(gd.view(np.uint32), rd.view(np.uint32))


@pytest.mark.parametrize("kind", ["sorted", "reversed", "lattice", "zero_rows", "tiny", "huge", "outlier"])
@pytest.mark.parametrize("metric", [0, 1, 2])
def test_graph_hard_values(kg, orc, kind, metric):
    rng = np.random.default_rng(7)
    x = rng.normal(0, 1, (1500, 12)).astype(np.float32)
    if kind in ("sorted", "reversed"):
        x = x[np.argsort(x[:, 0])][:: 1 if kind == "sorted" else -1] * 3
    elif kind == "lattice":
        x = rng.integers(-2, 3, (1500, 12)).astype(np.float32)
        x[700:900] = x[:200]
    elif kind == "zero_rows":
        x[::5] = 0
    elif kind == "tiny":
        x *= np.float32(1e-13)
    elif kind == "huge":
        x *= np.float32(1e18)
    else:
        x[17] *= np.float32(1e6)
    x = np.ascontiguousarray(x)
    gi, gd = kg.knn_graph(x, 25, metric=metric)
    ri, rd = orc.exact_knn(x, 25, threads=8) if metric == 2 else orc.exact_knn_metric(x, 25, metric, threads=8)
    assert np.array_equal(gi, ri)
    assert np.array_equal(gd.view(np.uint32), rd.view(np.uint32))


@pytest.mark.parametrize("n,d,k,folds,metric", [(256, 9, 32, 2, 2), (257, 16, 10, 10, 0), (700, 40, 31, 5, 1),
                                                (1281, 65, 20, 10, 2), (2600, 33, 5, 3, 0), (900, 12, 100, 10, 2)])
def test_fold_search_edges(kg, orc, n, d, k, folds, metric):
    x, y = datasets.gaussian_mixture(n=n, d=d, clusters=5, mean_scale=0.5, seed=n)
    a = kg.KNNCV(x, y, k=k, folds=folds, metric=metric, seed=4)
    b, fb, _ = orc.knncv(x, y, k=k, folds=folds, metric=metric, cv_seed=4)
    assert np.array_equal(a.fold_assignments, fb)
    assert np.array_equal(a.predicted_labels, b)


def test_resident_rows_off_alignment(kg):
    # a resident matrix that starts 4 bytes past a 16-byte boundary
    torch = pytest.importorskip("torch")
    x, _ = datasets.gaussian_mixture(n=900, d=16, seed=2)
    buf = torch.zeros(900 * 16 + 1, device="cuda")
    buf[1:] = torch.from_numpy(x).reshape(-1).cuda()
    torch.cuda.synchronize()
    kw = dict(runs=3, cycles=4, splitting=10, graph_neighbors=40, knn_k=8, materialize_graph=True)
    a = kg.KODAMA_matrix(buf[1:].view(900, 16), **kw)
    b = kg.KODAMA_matrix(x, **kw)
    assert np.array_equal(a.res, b.res)
    assert np.array_equal(a.knn_idx, b.knn_idx) and np.array_equal(a.knn_dist, b.knn_dist)
