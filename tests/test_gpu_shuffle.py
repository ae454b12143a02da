"""The group shuffle of the label evolution over the numbers of engine
regenerations (312 outputs, two positions a draw) that a shuffle runs through:
none, one, an odd or even number, block ends on and beside the last draw, odd and
even group counts.  Cycle after cycle the engine starts at another place in its
block.  A wrong position changes which rows are relabelled, so every result is
compared with the CPU restatement (std::shuffle's order) bit for bit, several
times over: the halves of the block that draw and place run side by side."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = [5, 6, 31, 64, 311, 312, 313, 620, 623, 624, 625, 626, 935, 936, 937, 1247, 1248, 1249, 1250, 1560, 1561,
          1872, 1875, 2000]


@pytest.mark.parametrize("groups", COUNTS)
def test_shuffled_proposals_match_oracle(kg, orc, groups):
    rng = np.random.default_rng(groups)
    k = min(4, groups - 1)
    gi, gd = orc.exact_knn(rng.standard_normal((groups, 3)).astype(np.float32), k, threads=4)
    labels = rng.integers(1, 4, groups).astype(np.int32)  # random: a flipped row shows in the next vote
    kw = dict(cycles=40, k=k, folds=2, index_base=0, cv_seed=3, stratified=False)
    for seed in (1, 2):
        a = orc.core_knn_graph(gi, gd, labels, evolutionary=True, guarded=False, absorption=False, seed=seed, **kw)
        for _ in range(3):
            b = kg.CoreKNNGraph(gi, gd, labels, evolutionary_search=True, guarded_diversity=False,
                                many_to_one_absorption=False, metric="euclidean", seed=seed, **kw)
            for f in ("clbest", "cvpredbest", "vect_acc", "vect_score", "proposal_size", "active_classes", "flags"):
                assert np.array_equal(getattr(b, f), getattr(a, f)), f
