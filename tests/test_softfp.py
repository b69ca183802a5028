"""The integer-pipe division and square root of the FP64 kernels
(csrc/softfp.cuh) against IEEE division and square root, bit for bit: random
and edge significands (all ones, powers of two, a few units around them),
quotients and squares next to representable and halfway values, zeros, and
exponents over the whole range, where the routines must either report that
the operands are outside theirs or be right.  On the CPU with seeds displaced
by MUFU's error bounds, on the GPU with MUFU itself."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "amr2d_mhd_gb300", "csrc")


def check_lib(gpu):
    src = os.path.join(HERE, "softfp_check.cu")
    out = os.path.join(HERE, "_build", "softfp_%s.so" % ("gpu" if gpu else "cpu"))
    if not os.path.exists(out) or os.path.getmtime(out) < max(os.path.getmtime(src),
                                                             os.path.getmtime(os.path.join(CSRC, "softfp.cuh"))):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        cmd = ([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-shared", "-Xcompiler", "-fPIC", "-gencode",
                "arch=compute_103a,code=sm_103a", "-fmad=false"] if gpu else
               ["g++", "-x", "c++", "-shared", "-fPIC", "-ffp-contract=off"])
        subprocess.check_call(cmd + ["-O2", "-std=c++17", "-I" + CSRC, src, "-o", out])
    L = ctypes.CDLL(out)
    L.softfp_check.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_double, ctypes.c_void_p,
                               ctypes.c_void_p]
    return L


def operands(n, seed):
    """n (a, b): significands and exponents of every kind the docstring names."""
    g = np.random.default_rng(seed)

    def mant():
        m = g.integers(0, 1 << 52, n, dtype=np.uint64)
        k = g.integers(0, 8, n)
        few, bit = m & 7, np.uint64(1) << (m % 52)
        ones = np.uint64((1 << 52) - 1)
        return np.select([k == 0, k == 1, k == 2, k == 3, k == 4, k == 5], [few, ones - few, bit, ones ^ bit,
                                                                            m & ~(bit - np.uint64(1)),
                                                                            m | (bit - np.uint64(1))], m)

    def num():
        e = np.where(g.random(n) < 0.8, g.integers(963, 1083, n), g.integers(0, 2048, n)).astype(np.uint64)
        s = g.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
        return (s | e << np.uint64(52) | mant()).view(np.float64)
    a, b = num(), num()
    with np.errstate(all="ignore"):
        pick = g.integers(0, 4, n)
        near = np.where(pick == 1, a * b, np.where(pick == 2, b * b, a))  # quotient near a, root near |b|
        near = (near.view(np.int64) + np.where(pick > 0, g.integers(-1, 2, n), 0)).view(np.float64)
    near[g.random(n) < 0.02] = 0.0
    near[g.random(n) < 0.02] = -0.0
    return near, b


def compare(L, n, seed, rel=0.0):
    a, b = operands(n, seed)
    out, bad = np.zeros((4, n)), np.zeros(n, np.uint8)
    assert L.softfp_check(a.ctypes.data, b.ctypes.data, n, rel, out.ctypes.data, bad.ctypes.data) == 0
    with np.errstate(all="ignore"):
        want = [a / b, np.sqrt(a), a / 3.0, a / 6.0]
    for k, w in enumerate(want):
        ok = (bad >> k & 1) == 0
        assert np.array_equal(out[k][ok].view(np.int64), w[ok].view(np.int64)), k
        # operands of ordinary size, and zeros, are never refused (sqrt: of either zero or positive numbers)
        with np.errstate(all="ignore"):
            mid = (np.abs(a) > 1e-150) & (np.abs(a) < 1e150) & (np.abs(b) > 1e-150) & (np.abs(b) < 1e150)
        mid |= (a == 0) & (np.abs(b) > 1e-300) & (np.abs(b) < 1e300)
        if k == 1:
            mid &= a >= 0
        assert ok[mid].all(), k


@pytest.mark.parametrize("rel", [0.0, 2.0 ** -22.9, -2.0 ** -22.9])
def test_soft_division_and_root_on_the_cpu(rel):
    compare(check_lib(False), 1 << 20, 7, rel)


@pytest.mark.gpu
def test_soft_division_and_root_on_the_gpu(gpu):
    L = check_lib(True)
    for seed in range(8):
        compare(L, 1 << 20, seed)


def compare_mul(L, n, seed):
    """Products and the conversions between double and float, bit for bit."""
    a, b = operands(n, seed)
    g = np.random.default_rng(seed + 1)
    few = g.random(n) < 0.3   # on float's grid and halfway between its values
    a[few] = (a[few].view(np.int64) & ~np.int64((1 << 28) - 1)).view(np.float64)
    out, bad = np.zeros((3, n)), np.zeros(n, np.uint8)
    L.softmul_check.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p, ctypes.c_void_p]
    assert L.softmul_check(a.ctypes.data, b.ctypes.data, n, out.ctypes.data, bad.ctypes.data) == 0
    ok = bad == 0
    with np.errstate(all="ignore"):
        p, f = a * b, a.astype(np.float32).astype(np.float64)
        mid = (np.abs(a) > 1e-150) & (np.abs(a) < 1e150) & (np.abs(b) > 1e-150) & (np.abs(b) < 1e150)
    assert np.array_equal(out[0][ok].view(np.int64), p[ok].view(np.int64))
    assert ok[mid].all() and ok[(a == 0) & np.isfinite(b) & (np.abs(b) > 1e-300)].all()
    for o in out[1:]:
        nan = np.isnan(f)
        assert np.array_equal(np.isnan(o), nan) and np.array_equal(o[~nan].view(np.int64), f[~nan].view(np.int64))


def test_soft_product_and_conversions_on_the_cpu():
    compare_mul(check_lib(False), 1 << 20, 21)


@pytest.mark.gpu
def test_soft_product_and_conversions_on_the_gpu(gpu):
    for seed in range(30, 34):
        compare_mul(check_lib(True), 1 << 20, seed)


@pytest.mark.gpu
@pytest.mark.parametrize("flux", ["RUSA", "HLLE", "HLLC", "HLLD"])
def test_riemann_with_operands_outside_the_soft_range(gpu, flux):
    """Face states with zero, subnormal, tiny and huge components, where the
    kernel falls back to the native operators, against the oracle bit for bit."""
    from oracle import pyoracle as P
    g = np.random.default_rng(11)
    n = 4000
    w = g.normal(0.0, 1.0, (2, n, 8))
    w[..., 0], w[..., 4] = g.uniform(0.1, 3.0, (2, n)), g.uniform(0.05, 2.0, (2, n))
    scale = g.choice([0.0, 1e-320, 1e-310, 1e-160, 1e-20, 1.0, 1.0, 1.0, 1e90], (2, n, 8))
    cols = [1, 2, 3, 5, 6, 7]
    w[..., cols] *= scale[..., cols]
    w[..., 4] *= g.choice([1e-300, 1e-20, 1.0, 1.0], (2, n))
    w[1, :, 5] = w[0, :, 5]
    out, st = gpu.riemann(flux, w[0], w[1], 5.0 / 3.0)
    names = ["RUSA", "HLLE", "HLLC", "HLLD"]
    want = np.zeros(8)
    for i in range(n):
        l, r = np.ascontiguousarray(w[0, i]), np.ascontiguousarray(w[1, i])
        rc = P.lib().oracle_riemann(names.index(flux), l.ctypes.data, r.ctypes.data, 5.0 / 3.0, 0, want.ctypes.data)
        assert (st[i] != 0) == (rc != 0), i
        if rc == 0:
            assert np.array_equal(out[i], want, equal_nan=True), (i, out[i], want)
