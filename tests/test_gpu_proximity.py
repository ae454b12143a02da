"""Co-label proximity at the edges of its kernel's splits (32 neighbours per
batch, 4 per step, label vectors of 4 ints shared by 8 lanes, and the unpadded
rows the allocation-free entry point falls back to) against the CPU
restatement, bit for bit: both form the same integer counts and the same
double-rounded arithmetic, so the tolerance is 0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n, K, runs):
    rng = np.random.default_rng(n * 1000 + K * 10 + runs)
    idx = rng.integers(1, n + 1, (n, K)).astype(np.int32)
    idx[rng.random((n, K)) < 0.05] = -1
    dist = (rng.random((n, K), dtype=np.float32) * 4.0 - 0.25).astype(np.float32)
    dist[rng.random((n, K)) < 0.02] = np.inf
    dist[:, ::7] = dist[:, :1]  # tied distances: the id decides
    return idx, dist, rng.integers(0, 4, (runs, n)).astype(np.int32)


@pytest.mark.parametrize("n,K,runs", [(3, 1, 1), (9, 4, 3), (33, 31, 4), (100, 33, 37), (65, 100, 32), (257, 130, 131),
                                      (4194240, 1, 1)])
def test_proximity_edges(kg, orc, n, K, runs):
    torch = pytest.importorskip("torch")
    idx, dist, res = _case(n, K, runs)
    want_i, want_d = orc.dissimilarity(idx, dist, res)
    host_i, host_d = idx.copy(), dist.copy()
    kg.KODAMADissimilarityInPlace(host_i, host_d, res)
    dev_i, dev_d = torch.from_numpy(idx).cuda(), torch.from_numpy(dist).cuda()
    kg.KODAMADissimilarityInPlace_device(dev_i, dev_d, torch.from_numpy(res).cuda())
    for name, gi, gd in (("host", host_i, host_d), ("device", dev_i.cpu().numpy(), dev_d.cpu().numpy())):
        assert np.array_equal(gi, want_i), name
        assert np.array_equal(gd.view(np.uint32), want_d.view(np.uint32)), name
