"""The neighbour search where the device has no room for the tensor search's candidate
lists: the brute force takes the call, with the same graph."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# in a process of its own, whose memory pool is empty: 120000 rows and 200 neighbours take
# 2.75 GB of scratch, 0.77 GB by the brute force
SCRIPT = """
import numpy as np, torch
import kodama_gb300 as kg
x = np.random.default_rng(5).standard_normal((120000, 2)).astype(np.float32)
kg.knn_graph(x[:2000], 200)
free = torch.cuda.mem_get_info()[0]
hold = torch.empty(free - (2 << 30), dtype=torch.uint8, device="cuda")
a = kg.knn_graph(x, 200, return_fallback=True)
assert a[2] == 120000, a[2]
del hold
torch.cuda.empty_cache()
b = kg.knn_graph(x, 200, return_fallback=True)
assert b[2] < 120000, b[2]
assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
print("same")
"""


def test_graph_without_room_for_the_lists(kg):
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout + r.stderr
