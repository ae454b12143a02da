"""The graph's choice between the tensor search and the brute force (knn_tc_pays): few
rows, few neighbours, many coordinates, points on a line or a circle.  On both sides
of the rule the graph is the CPU restatement's, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,K,metric", [
    (97, 65, 5, 1), (97, 3, 96, 0), (97, 3, 10, 2), (100, 100, 30, 2), (128, 256, 1, 0), (200, 70, 40, 1), (255, 64, 1, 2),
    (255, 64, 20, 2), (255, 2, 90, 0), (256, 8, 1, 0), (512, 16, 5, 1), (512, 16, 7, 1), (1000, 4, 2, 0), (1000, 4, 5, 0),
    (2000, 2, 1, 2), (4000, 2, 1, 2), (9001, 1, 3, 2), (9001, 1, 4, 2), (9001, 2, 2, 0), (9001, 2, 20, 0), (9001, 1, 5, 1)])
def test_graph_on_both_sides(kg, orc, n, d, K, metric):
    x = np.random.default_rng(n + d).standard_normal((n, d)).astype(np.float32)
    gi, gd = kg.knn_graph(x, K, metric=metric)
    ri, rd = orc.exact_knn(x, K, threads=8) if metric == 2 else orc.exact_knn_metric(x, K, metric, threads=8)
    assert np.array_equal(gi, ri)
    assert np.array_equal(gd.view(np.uint32), rd.view(np.uint32))


# the rows the brute force computed: all of them where it is the faster way
@pytest.mark.parametrize("n,d,K,tensor", [
    (100, 100, 30, True), (100, 8, 30, True), (256, 8, 1, False), (256, 8, 10, True), (1000, 8, 1, False),
    (1000, 100, 1, True), (8000, 8, 1, True), (30000, 1, 10, False)])
def test_route(kg, n, d, K, tensor):
    x = np.random.default_rng(n).standard_normal((n, d)).astype(np.float32)
    rows = kg.knn_graph(x, K, return_fallback=True)[2]
    assert (rows < n) == tensor
