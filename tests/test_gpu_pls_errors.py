"""PLS-LDA calls that end in an error on the device: a pooled covariance that is not
positive definite (every row a class of its own in tight clusters) and a fit without a
direction (constant columns).  Steps queued behind the failing evaluation take its
predictions as class codes, so these have to be codes; the call reports the
reference's error and the next one is answered as ever."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clusters(n, p, c, seed):
    r = np.random.default_rng(seed)
    lab = r.integers(0, c, n)
    return (r.standard_normal((n, p)) + 4 * r.standard_normal((c, p))[lab]).astype(np.float32), r


def _healthy(kg, orc):
    x, r = _clusters(200, 6, 3, 7)
    lab = r.integers(1, 5, 200).astype(np.int32)
    a = orc.core_plslda(x, lab, components=2, cycles=3, folds=4, stratified=False, guarded=True, absorption=True,
                        evolutionary=True, seed=1, cv_seed=2)
    b = kg.CorePLSLDA(x, lab, max_components=2, fixed_components=2, cycles=3, folds=4, stratified=False,
                      guarded_diversity=True, many_to_one_absorption=True, evolutionary_search=True, seed=1, cv_seed=2)
    assert np.array_equal(b.clbest, a.clbest) and np.array_equal(b.vect_score, a.vect_score)


@pytest.mark.parametrize("n,p", [(60, 8), (75, 12), (400, 20)])
@pytest.mark.parametrize("coarsening", [False, True])
def test_singular_covariance(kg, orc, n, p, coarsening):
    x, r = _clusters(n, p, 4, n)
    lab = (r.permutation(n) + 1).astype(np.int32)
    kw = dict(cycles=5, folds=10, stratified=False, seed=3, cv_seed=4)
    with pytest.raises(RuntimeError, match="Cholesky"):
        orc.core_plslda(x, lab, components=p, guarded=True, absorption=True, coarsening=coarsening, **kw)
    for _ in range(3):
        with pytest.raises(RuntimeError, match="Cholesky"):
            kg.CorePLSLDA(x, lab, max_components=p, fixed_components=p, guarded_diversity=True,
                          many_to_one_absorption=True, auto_class_coarsening=coarsening, **kw)
    _healthy(kg, orc)


def test_an_early_failure_is_not_forgotten(kg, orc):
    # the first evaluation fails; absorption and coarsening would mend the later ones
    for n, p, c in ((120, 5, 3), (80, 4, 2)):
        x, r = _clusters(n, p, c, n)
        lab = (r.permutation(n) + 1).astype(np.int32)
        kw = dict(cycles=30, folds=5, stratified=False, seed=3, cv_seed=4)
        with pytest.raises(RuntimeError, match="Cholesky"):
            orc.core_plslda(x, lab, components=p, guarded=True, absorption=True, coarsening=True, evolutionary=True, **kw)
        with pytest.raises(RuntimeError, match="Cholesky"):
            kg.CorePLSLDA(x, lab, max_components=p, fixed_components=p, guarded_diversity=True, evolutionary_search=True,
                          many_to_one_absorption=True, auto_class_coarsening=True, **kw)
    _healthy(kg, orc)


def test_singular_covariance_in_a_matrix(kg, orc):
    x, r = _clusters(300, 10, 5, 1)
    start = (r.permutation(300) + 1).astype(np.int32)
    for _ in range(3):
        with pytest.raises(RuntimeError, match="Cholesky"):
            kg.KODAMA_matrix(x, runs=4, cycles=4, classifier="pls", components=10, graph_neighbors=10, knn_k=5, folds=5,
                             starting_labels=start)
    _healthy(kg, orc)


def test_no_direction(kg, orc):
    x = np.full((80, 5), 2.5, np.float32)
    lab = (np.arange(80) % 4 + 1).astype(np.int32)
    with pytest.raises(RuntimeError, match="no supervised latent direction"):
        orc.plsldapredict(x[:50], lab[:50], x[50:], components=2)
    for _ in range(3):
        with pytest.raises(RuntimeError, match="no supervised latent direction"):
            kg.PLSLDAPredict(x[:50], lab[:50], x[50:], max_components=2, fixed_components=2)
    _healthy(kg, orc)
