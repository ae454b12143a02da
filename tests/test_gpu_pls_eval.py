"""PLS-LDA evaluation at the sizes where its split changes: widths around the
16-feature blocks and the 4-float pitch, row counts around the 32-row batches and
the 4096 from which a warp follows the scores, one to eight components, more
classes than the streamed cross-products hold sums for, and constant columns.
Every chain keeps the CPU restatement's order, so results are equal bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, p, classes, seed):
    rng = np.random.default_rng(seed)
    lab = rng.integers(1, classes + 1, n).astype(np.int32)
    x = rng.standard_normal((n, p)) + 0.8 * rng.standard_normal((classes + 1, p))[lab]
    return x.astype(np.float32), lab


@pytest.mark.parametrize("n,p,classes,comp,folds,da", [
    (33, 3, 2, 1, 3, False), (64, 16, 3, 2, 2, False), (97, 17, 4, 3, 5, False), (257, 31, 5, 7, 4, False),
    (300, 33, 6, 8, 4, False), (511, 12, 40, 4, 3, True), (4095, 18, 7, 5, 2, False), (4097, 20, 7, 5, 2, False),
    (4500, 47, 9, 7, 3, False), (4200, 14, 5, 6, 2, True), (4000, 10, 1600, 2, 2, False),
])
def test_evaluation_matches_oracle(kg, orc, n, p, classes, comp, folds, da):
    x, lab = _data(n, p, classes, seed=n + p)
    x[:, p // 2] = 3.25  # no variance: a column of zeros
    kw = dict(folds=folds, stratified=False, max_components=comp, fixed_components=comp, cv_seed=5)
    pred, fo, sel, abc, _ = orc.plsldacv(x, lab, da=da, **kw)
    g = (kg.PLSDACV if da else kg.PLSLDACV)(x, lab, **kw)
    assert np.array_equal(g.fold_assignments, fo)
    assert np.array_equal(g.predicted_labels, pred) and g.selected_components == sel


@pytest.mark.parametrize("n,p,classes,comp", [(500, 19, 30, 3), (4600, 21, 40, 5)])
def test_core_matches_oracle(kg, orc, n, p, classes, comp):
    # the Gram evaluations (from the second cycle on)
    x, lab = _data(n, p, classes, seed=n)
    x[:, 1] = 0.0
    con = np.arange(1, n + 1, dtype=np.int32)
    kw = dict(cycles=4, folds=3, stratified=False, evolutionary=True, guarded=True, absorption=True,
              coarsening=True, seed=11, cv_seed=12)
    a = orc.core_plslda(x, lab, constrain=con, fixed=None, components=comp, **kw)
    b = kg.CorePLSLDA(x, lab, constrain=con, cycles=4, folds=3, stratified=False, max_components=comp,
                      fixed_components=comp, evolutionary_search=True, guarded_diversity=True,
                      many_to_one_absorption=True, auto_class_coarsening=True, seed=11, cv_seed=12)
    assert np.array_equal(b.clbest, a.clbest)
    assert np.array_equal(b.cvpredbest, a.cvpredbest)
    assert np.array_equal(b.vect_score, a.vect_score)
