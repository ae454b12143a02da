"""The rounds of a PLS-LDA evaluation whose score cross-products follow the scores (from
4096 rows on): fifteen warps score batches of 64 rows (32 with one component) while one
follows a round behind.  Row counts on, beside and short of whole rounds and batches,
with and without the fold Gram.  Results equal the CPU restatement's bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, p, classes, seed):
    rng = np.random.default_rng(seed)
    lab = rng.integers(1, classes + 1, n).astype(np.int32)
    x = rng.standard_normal((n, p)) + 0.8 * rng.standard_normal((classes + 1, p))[lab]
    return x.astype(np.float32), lab


@pytest.mark.parametrize("n,comp", [(4096, 1), (4096, 7), (4320, 1), (4321, 1), (4799, 3), (4800, 3), (4801, 3),
                                    (5696, 4), (5760, 4), (5761, 4), (6000, 8)])
def test_rounds_match_oracle(kg, orc, n, comp):
    x, lab = _data(n, 11, 5, n + comp)
    kw = dict(folds=2, stratified=False, max_components=comp, fixed_components=comp, cv_seed=5)
    pred, fo, sel, _, _ = orc.plsldacv(x, lab, da=False, **kw)
    g = kg.PLSLDACV(x, lab, **kw)
    assert np.array_equal(g.fold_assignments, fo)
    assert np.array_equal(g.predicted_labels, pred) and g.selected_components == sel


@pytest.mark.parametrize("n,comp", [(4800, 2), (5761, 7)])
def test_rounds_with_gram_match_oracle(kg, orc, n, comp):
    x, lab = _data(n, 13, 9, n + comp)
    con = np.arange(1, n + 1, dtype=np.int32)
    kw = dict(cycles=3, folds=2, stratified=False, seed=11, cv_seed=12)
    a = orc.core_plslda(x, lab, constrain=con, fixed=None, components=comp, evolutionary=True, guarded=True,
                        absorption=True, coarsening=True, **kw)
    b = kg.CorePLSLDA(x, lab, constrain=con, max_components=comp, fixed_components=comp, evolutionary_search=True,
                      guarded_diversity=True, many_to_one_absorption=True, auto_class_coarsening=True, **kw)
    assert np.array_equal(b.clbest, a.clbest)
    assert np.array_equal(b.cvpredbest, a.cvpredbest)
    assert np.array_equal(b.vect_score, a.vect_score)
