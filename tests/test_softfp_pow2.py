"""Products with powers of two on the exponent field (scale_pow2 and times_pow2
of csrc/softfp.cuh) against IEEE products, bit for bit, over the whole range of
exponents and densest at its ends: either the routine reports that operand or
result are outside the normal range, or it is right; it never refuses what is
well inside, nor a zero."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "amr2d_mhd_gb300", "csrc")


def check_lib(gpu):
    src = os.path.join(HERE, "softfp_pow2_check.cu")
    out = os.path.join(HERE, "_build", "softfp_pow2_%s.so" % ("gpu" if gpu else "cpu"))
    if not os.path.exists(out) or os.path.getmtime(out) < max(os.path.getmtime(src),
                                                             os.path.getmtime(os.path.join(CSRC, "softfp.cuh"))):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        cmd = ([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-shared", "-Xcompiler", "-fPIC", "-gencode",
                "arch=compute_103a,code=sm_103a", "-fmad=false"] if gpu else
               ["g++", "-x", "c++", "-shared", "-fPIC", "-ffp-contract=off"])
        subprocess.check_call(cmd + ["-O2", "-std=c++17", "-I" + CSRC, src, "-o", out])
    L = ctypes.CDLL(out)
    L.pow2_check.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p, ctypes.c_void_p]
    return L


def compare(L, seed, n=1 << 20):
    g = np.random.default_rng(seed)
    ends = np.concatenate([np.arange(0, 8), np.arange(2040, 2048)])
    e = np.where(g.random(n) < 0.5, g.choice(ends, n), g.integers(0, 2048, n)).astype(np.uint64)
    m = g.integers(0, 1 << 52, n, dtype=np.uint64)
    m[g.random(n) < 0.1] = 0
    x = (g.integers(0, 2, n, dtype=np.uint64) << np.uint64(63) | e << np.uint64(52) | m).view(np.float64)
    x[g.random(n) < 0.02] = 0.0
    x[g.random(n) < 0.02] = -0.0
    k = np.where(g.random(n) < 0.5, g.integers(1, 2047, n), g.integers(1018, 1029, n)).astype(np.uint64)
    p = (k << np.uint64(52)).view(np.float64)
    out, bad = np.zeros((5, n)), np.zeros(n, np.uint8)
    assert L.pow2_check(x.ctypes.data, p.ctypes.data, n, out.ctypes.data, bad.ctypes.data) == 0
    with np.errstate(all="ignore"):
        want = [0.25 * x, 0.5 * x, 2.0 * x, 4.0 * x, x * p]
        inside = (np.abs(x) > 1e-290) & (np.abs(x) < 1e290)
        for q, w in enumerate(want):
            ok = (bad >> q & 1) == 0
            assert np.array_equal(out[q][ok].view(np.int64), w[ok].view(np.int64)), q
            sure = (x == 0) | (inside & (np.abs(w) > 1e-290) & (np.abs(w) < 1e290))
            assert ok[sure].all(), q


def test_powers_of_two_on_the_cpu():
    compare(check_lib(False), 3)


@pytest.mark.gpu
def test_powers_of_two_on_the_gpu(gpu):
    for seed in range(4):
        compare(check_lib(True), seed)
