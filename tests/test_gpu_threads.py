"""Calls of several host threads whose kernels are the same but whose shared-memory
sizes are not: every call's results are those of a call by itself."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hammer(calls, rounds):
    want = [c() for c in calls]
    errors = []

    def work(i):
        try:
            for _ in range(rounds):
                got = calls[i]()
                if not all(np.array_equal(a, b) for a, b in zip(got, want[i])):
                    raise AssertionError("call %d: other results" % i)
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_graphs_of_several_threads(kg):
    rng = np.random.default_rng(0)
    xs = [rng.standard_normal((n, d)).astype(np.float32) for n, d in ((300, 8), (700, 256), (400, 40), (600, 200))]
    _hammer([lambda x=x: kg.knn_graph(x, 20, metric="euclidean") for x in xs], 150)


def test_evolutions_of_several_threads(kg):
    rng = np.random.default_rng(1)
    calls = []
    for n, classes, p in ((300, 4, 12), (1500, 60, 30), (800, 200, 5)):
        x = rng.standard_normal((n, p)).astype(np.float32)
        lab = rng.integers(1, classes + 1, n).astype(np.int32)

        def knn(x=x, lab=lab):
            r = kg.CoreKNN(x, lab, cycles=4, folds=4, k=6, metric="euclidean", stratified=False)
            return r.clbest, r.vect_score

        def pls(x=x, lab=lab):
            r = kg.CorePLSLDA(x, lab, cycles=2, folds=3, stratified=False, max_components=3, fixed_components=3)
            return r.clbest, r.vect_score

        calls += [knn, pls]
    _hammer(calls, 25)


def test_matrices_of_several_threads(kg):
    rng = np.random.default_rng(2)
    calls = []
    for n, d, split in ((400, 6, 20), (900, 40, 60), (700, 90, 150)):
        x = rng.standard_normal((n, d)).astype(np.float32)

        def call(x=x, split=split):
            r = kg.KODAMA_matrix(x, runs=3, cycles=3, splitting=split, graph_neighbors=12, knn_k=6)
            return r.res, r.acc

        calls.append(call)
    _hammer(calls, 25)
