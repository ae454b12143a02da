"""The loadings of a PLS component (block_loading, exact_dot.cuh) against the sequential
double sums they stand for, rounded to float: columns from the smallest normal values,
whose products lose their remainders to underflow, over ordinary ones to large ones,
with row counts on and beside the chunks of eight and of 1024 rows.  Equal bit for
bit."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pls_loading") / "libpls_loading_probe.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                    "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-I",
                    os.path.join(ROOT, "kodama_gb300", "csrc"), "-o", out,
                    os.path.join(HERE, "probes", "pls_loading_probe.cu")], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("n,p", [(3, 512), (8, 1024), (9, 1000), (63, 513), (64, 1024), (300, 700), (1025, 511), (2049, 64)])
def test_loadings_are_the_sequential_sums(probe, n, p):
    rng = np.random.default_rng(n + p)
    zp = (p + 7) // 8 * 8
    scale = 2.0 ** np.resize([-116, 0, -112, -120, -60, -118, -100, -116, 20, -122], p)
    z = np.zeros((n, zp), np.float32)
    z[:, :p] = rng.standard_normal((n, p)) * scale
    sc = (rng.standard_normal(n) / np.sqrt(n)).astype(np.float32)
    top = ((z.view(np.uint32) >> 23) & 0xff).max(axis=0)
    zexp = np.maximum(top[:p], 1).astype(np.int32)
    want = np.zeros(p)
    for i in range(n):  # the chain: exact products, one rounding an addition
        want += z[i, :p].astype(np.float64) * np.float64(sc[i])
    got = np.zeros(p, np.float32)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert probe.loading_probe(ptr(z), zp, p, n, ptr(sc), ptr(zexp), ptr(got)) == 0
    assert np.array_equal(got.view(np.uint32), want.astype(np.float32).view(np.uint32))
