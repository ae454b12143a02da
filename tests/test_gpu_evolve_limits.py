"""Label evolution at the sizes where its kernels change: rows around the 1024
threads and 8-row vectors, few to very many labels, counters for all warps, a few
or one, rows in shared or global memory, neighbour lists of every
width, equal distances (exact ties of the votes) and rows whose neighbours all
share their fold.  The CPU restatement's results are equal bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("folds", "clbest", "cvpredbest", "vect_acc", "vect_score", "proposal_size", "active_classes", "flags")


def _same(b, a):
    for f in FIELDS:
        assert np.array_equal(getattr(b, "fold_assignments" if f == "folds" else f), getattr(a, f)), f
    n = len(a.counters)
    assert np.array_equal(b.counters[:n], a.counters)


@pytest.mark.parametrize("n,classes,w,folds,cycles", [
    (9, 3, 3, 3, 6), (33, 33, 8, 5, 10), (1023, 40, 1, 4, 12), (1024, 2, 9, 4, 12), (1025, 100, 16, 7, 12),
    (2050, 33, 30, 10, 12), (5000, 300, 32, 10, 10),
    (15001, 60, 10, 5, 6),   # rows in global memory
    (2400, 2400, 5, 4, 4),   # counters for a few warps
    (3670, 3670, 5, 4, 3),   # counters for one
])
def test_knn_evolution_matches_oracle(kg, orc, n, classes, w, folds, cycles):
    rng = np.random.default_rng(n)
    x = rng.integers(0, 12, (n, 3)).astype(np.float32)  # a lattice: many equal distances
    g = min(n - 1, max(w, 2))
    gi, gd = orc.exact_knn(x, g, threads=8)
    labels = (np.arange(n) % classes + 1).astype(np.int32)
    rng.shuffle(labels)
    kw = dict(cycles=cycles, k=w, folds=folds, index_base=0, seed=5, cv_seed=6, stratified=False)
    for evo, ab in ((True, True), (False, False)):
        a = orc.core_knn_graph(gi, gd, labels, evolutionary=evo, guarded=True, absorption=ab, **kw)
        b = kg.CoreKNNGraph(gi, gd, labels, evolutionary_search=evo, guarded_diversity=True,
                            many_to_one_absorption=ab, metric="euclidean", **kw)
        _same(b, a)


@pytest.mark.parametrize("n,classes,co,fixed", [(1125, 100, True, False), (1031, 33, True, True), (40, 12, True, False)])
def test_pls_evolution_matches_oracle(kg, orc, n, classes, co, fixed):
    rng = np.random.default_rng(n)
    labels = rng.integers(1, classes + 1, n).astype(np.int32)
    x = (rng.standard_normal((n, 12)) + 0.8 * rng.standard_normal((classes + 1, 12))[labels]).astype(np.float32)
    con = np.arange(1, n + 1, dtype=np.int32)
    fix = (rng.random(n) < 0.05).astype(np.int32) if fixed else None
    kw = dict(cycles=10, folds=4, stratified=False, seed=11, cv_seed=12)
    a = orc.core_plslda(x, labels, constrain=con, fixed=fix, components=3, evolutionary=True, guarded=True,
                        absorption=True, coarsening=co, **kw)
    b = kg.CorePLSLDA(x, labels, constrain=con, fixed=fix, max_components=3, fixed_components=3,
                      evolutionary_search=True, guarded_diversity=True, many_to_one_absorption=True,
                      auto_class_coarsening=co, **kw)
    _same(b, a)
