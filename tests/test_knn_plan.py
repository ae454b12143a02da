"""Host-side plans of the tensor-core neighbour search (knn_tc.cu), without a GPU:
the scratch at row counts whose tile pairs pass 2^31 and 2^32, the fold plan's
layout, and its rule at fold counts where padding costs too much."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    from kodama_gb300 import build as kbuild
    lib = kbuild.build()
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")))
    out = str(tmp_path_factory.mktemp("knn_plan") / "libknn_plan_probe.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "kodama_gb300", "csrc"),
                    "-I", os.path.join(cuda, "include"), os.path.join(HERE, "probes", "knn_plan_probe.cpp"),
                    "-o", out, "-L", os.path.dirname(lib), "-lkodama_gb300", "-Wl,-rpath," + os.path.dirname(lib)],
                   check=True)
    p = ctypes.CDLL(out)
    p.probe_scratch.restype = ctypes.c_longlong
    return p


# rows x 4 KB of lists (128 entries, two segments and two groups), and under 1 KB a row
# of operands, copies and the brute force's room beside them
@pytest.mark.parametrize("n", [1_000_000, 8_388_608, 8_388_609, 11_900_000, 20_000_000, 1 << 26])
def test_scratch_grows_with_the_rows(probe, n):
    assert probe.probe_supported(n, 10, 10)
    assert 4096 * n <= probe.probe_scratch(n, 10, 10, 152) < 5120 * n


def test_row_limit(probe):
    assert not probe.probe_supported((1 << 26) + 1, 10, 10)


@pytest.mark.parametrize("n,d,K,metric,tensor", [
    (96, 100, 30, 2, False), (100, 100, 30, 2, True), (256, 8, 1, 0, False), (256, 8, 10, 0, True), (1 << 25, 50, 30, 2, True),
    (30000, 1, 10, 2, False), (30000, 1, 11, 2, True), (30000, 2, 10, 0, False), (30000, 2, 10, 1, True), (1000, 257, 5, 2, False)])
def test_graph_rule(probe, n, d, K, metric, tensor):
    assert bool(probe.probe_pays(n, d, K, metric)) == tensor


def _plan(probe, folds, d, K):
    n = len(folds)
    folds = np.ascontiguousarray(folds, np.int32)
    pairs = ctypes.c_int()
    tiles = probe.probe_fold_plan(folds.ctypes.data_as(ctypes.c_void_p), n, d, K, None, None, None,
                                  ctypes.byref(pairs))
    if tiles == 0:
        return None
    perm, off, skip = np.zeros(tiles * 256, np.int32), np.zeros(2 * tiles, np.int32), np.zeros((2 * tiles, 2), np.int32)
    assert probe.probe_fold_plan(folds.ctypes.data_as(ctypes.c_void_p), n, d, K, perm.ctypes.data_as(ctypes.c_void_p),
                                 off.ctypes.data_as(ctypes.c_void_p), skip.ctypes.data_as(ctypes.c_void_p),
                                 ctypes.byref(pairs)) == tiles
    return perm, off, skip, pairs.value


@pytest.mark.parametrize("n,folds", [(1000, 2), (1000, 10), (4096, 7), (20000, 100)])
def test_fold_plan_layout(probe, n, folds):
    f = np.random.default_rng(n).integers(0, folds, n)
    f[f == 1] = 0  # a fold number that does not occur
    perm, off, skip, pairs = _plan(probe, f, 50, 30)
    tiles = len(perm) // 256
    assert np.array_equal(np.sort(perm[perm >= 0]), np.arange(n))
    at = 0
    for q in range(2 * tiles):
        rows = perm[q * 128:(q + 1) * 128]
        rows = rows[rows >= 0]
        assert off[q] == at
        if len(rows) == 0:
            assert skip[q, 1] == tiles
            continue
        first, count = skip[q]
        own = perm[first * 256:(first + count) * 256]
        assert len(set(f[rows])) == 1 and np.array_equal(own[own >= 0], np.flatnonzero(f == f[rows[0]]))
        at += tiles - count
    assert pairs == at


@pytest.mark.parametrize("n,d,K,folds,tensor", [
    (10000, 50, 10, 10, True), (10000, 50, 10, 100, True), (10000, 50, 10, 10000, False), (10000, 128, 10, 10000, False),
    (1000, 50, 100, 200, True), (1000, 8, 10, 500, False), (46400, 1, 1, 46400, False), (65535, 256, 200, 65535, False)])
def test_fold_plan_rule(probe, n, d, K, folds, tensor):
    assert (_plan(probe, np.arange(n) % folds, d, K) is not None) == tensor
