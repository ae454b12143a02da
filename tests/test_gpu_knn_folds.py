"""KNNCV and CoreKNN with many folds, on both sides of the rule between the tensor
search, which pads every fold to whole tiles, and the brute force: leave-one-out,
hundreds of small folds, folds of uneven sizes, more folds asked for than rows.  The
CPU restatement's results are equal bit for bit."""

import numpy as np
import pytest

from kodama_gb300 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,folds,metric,stratified", [
    (300, 5, 1, 300, 2, False), (300, 70, 20, 150, 2, False), (1001, 9, 10, 60, 2, False), (1001, 9, 10, 70, 0, False),
    (1001, 9, 100, 300, 2, True), (1500, 66, 7, 400, 1, False), (1500, 66, 7, 1500, 2, False), (2050, 3, 3, 2050, 2, False),
    (4001, 12, 30, 200, 2, False), (4001, 12, 30, 2000, 0, True), (700, 8, 5, 5000, 2, True)])
def test_many_folds_match_oracle(kg, orc, n, d, k, folds, metric, stratified):
    x, y = datasets.gaussian_mixture(n=n, d=d, clusters=5, mean_scale=0.5, seed=n)
    a = kg.KNNCV(x, y, k=k, folds=folds, metric=metric, seed=4, stratified=stratified)
    b, fb, _ = orc.knncv(x, y, k=k, folds=folds, metric=metric, cv_seed=4, stratified=stratified)
    assert np.array_equal(a.fold_assignments, fb)
    assert np.array_equal(a.predicted_labels, b)


def test_uneven_groups_match_oracle(kg, orc):
    # constrained rows stay together: one fold of half the rows, many of one to four
    n = 1203
    x, y = datasets.gaussian_mixture(n=n, d=6, clusters=4, mean_scale=0.5, seed=3)
    con = np.concatenate([np.full(600, 1), 2 + np.arange(n - 600) // 4]).astype(np.int32)
    a = kg.KNNCV(x, y, constrain=con, k=8, folds=140, metric=2, seed=9, stratified=False)
    b, fb, _ = orc.knncv(x, y, constrain=con, k=8, folds=140, metric=2, cv_seed=9, stratified=False)
    assert np.array_equal(a.fold_assignments, fb)
    assert np.array_equal(a.predicted_labels, b)


def test_leave_one_out_of_many_rows(kg):
    """More folds than a 32-bit count of tile pairs holds.  Points on a line at whole
    numbers: the nearest is the neighbour across the smaller gap, the lower row of two
    equal ones."""
    n = 46400
    rng = np.random.default_rng(2)
    gap = rng.integers(1, 40, n - 1)
    x = np.concatenate([[0], np.cumsum(gap)]).astype(np.float32)[:, None]
    y = rng.integers(1, 9, n).astype(np.int32)
    left = np.concatenate([[10**9], gap])
    right = np.concatenate([gap, [10**9]])
    near = np.where(left <= right, np.arange(n) - 1, np.arange(n) + 1)
    r = kg.KNNCV(x, y, k=1, folds=n, metric="euclidean", seed=1, stratified=False)
    assert len(np.unique(r.fold_assignments)) == n
    assert np.array_equal(r.predicted_labels, y[near])
