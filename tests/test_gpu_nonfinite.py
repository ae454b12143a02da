"""Rows with infinite or missing values: every call ends, with labels of the input, and
the next one is answered as ever.  With one infinite row no distance is missing, so the
results are the CPU restatement's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, d, seed):
    r = np.random.default_rng(seed)
    lab = r.integers(1, 5, n).astype(np.int32)
    return (r.standard_normal((n, d)) + 1.5 * r.standard_normal((5, d))[lab]).astype(np.float32), lab


@pytest.mark.parametrize("n", [60, 700])
@pytest.mark.parametrize("metric", ["euclidean", "cosine", "inner_product"])
def test_one_infinite_row(kg, orc, n, metric):
    x, lab = _data(n, 6, n)
    if metric == "euclidean":
        x[7, 2] = np.inf
    m = ("cosine", "inner_product", "euclidean").index(metric)
    kw = dict(cycles=8, k=9, folds=4, stratified=False, seed=2, cv_seed=3)
    a = orc.core_knn(x, lab, metric=m, evolutionary=True, guarded=True, absorption=True, **kw)
    b = kg.CoreKNN(x, lab, metric=metric, evolutionary_search=True, guarded_diversity=True, many_to_one_absorption=True,
                   **kw)
    assert np.array_equal(b.clbest, a.clbest) and np.array_equal(b.vect_score, a.vect_score)


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("n,rows", [(60, 3), (700, 40), (700, 700)])
def test_missing_values(kg, orc, value, n, rows):
    x, lab = _data(n, 6, n)
    x[np.random.default_rng(1).permutation(n)[:rows], 2] = value
    for metric in ("euclidean", "cosine", "inner_product"):
        r = kg.CoreKNN(x, lab, metric=metric, cycles=6, k=9, folds=4, stratified=False, evolutionary_search=True,
                       guarded_diversity=True, many_to_one_absorption=True)
        assert np.isin(r.clbest, lab).all() and np.isin(r.cvpredbest, lab).all()
        assert np.isin(kg.KNNCV(x, lab, k=7, folds=4, metric=metric).predicted_labels, lab).all()
        gi, _ = kg.knn_graph(x, 12, metric=metric)
        assert gi.min() >= 0 and gi.max() < n
        m = kg.KODAMA_matrix(x, runs=3, cycles=4, splitting=8, graph_neighbors=12, knn_k=6, folds=3, metric=metric)
        assert m.res.min() >= 1
    for call in (lambda: kg.PLSLDACV(x, lab, folds=3, max_components=3, fixed_components=3).predicted_labels,
                 lambda: kg.CorePLSLDA(x, lab, cycles=3, folds=3, max_components=3, fixed_components=3,
                                       guarded_diversity=True, many_to_one_absorption=True).clbest):
        try:
            assert np.isin(call(), lab).all()
        except RuntimeError as e:
            assert "Cholesky" in str(e)
    y, lab2 = _data(200, 5, 9)
    kw = dict(cycles=5, k=5, folds=3, stratified=False, seed=2, cv_seed=3)
    a = orc.core_knn(y, lab2, metric=2, evolutionary=True, guarded=True, absorption=True, **kw)
    b = kg.CoreKNN(y, lab2, metric="euclidean", evolutionary_search=True, guarded_diversity=True,
                   many_to_one_absorption=True, **kw)
    assert np.array_equal(b.clbest, a.clbest)
