"""The FP32 path's pressure recovery as compiled, with the flags of the kernels
that use it (IEEE division; approximate division and FMA contraction), against
an evaluation in extended precision.  With 1/rho good to 2 ulp, its correction
leaves 2^-44 of |m|^2/rho, and the pairs' own error is below that: 2^-43 of the
subtracted terms and half a unit of the result, the bound of the same pairs
summed in FP64.  Where the terms cancel to the last bits of E, so that the
result's own rounding (2^-48 of the terms at most) does not hide it, the error is
compared with that form's: the additional errors are below 2^-53 of the terms,
1/16 of the pairs' 2^-49."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "amr2d_mhd_gb300", "csrc")
FLAGS = {"ieee": ["-fmad=false"], "fast": ["-prec-div=false", "-prec-sqrt=false"]}


def check_lib(name):
    src = os.path.join(HERE, "fp32_pressure_check.cu")
    out = os.path.join(HERE, "_build", "fp32_pressure_%s.so" % name)
    inputs = [src] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    if not os.path.exists(out) or os.path.getmtime(out) < max(os.path.getmtime(f) for f in inputs):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        subprocess.check_call([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-shared", "-Xcompiler", "-fPIC",
                               "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I" + CSRC]
                              + FLAGS[name] + [src, "-o", out])
    L = ctypes.CDLL(out)
    L.fp32_pressure.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p]
    return L


def states(n, seed, cancel):
    g = np.random.default_rng(seed)
    rho = 10.0 ** g.uniform(-3, 3, n)
    v = g.standard_normal((3, n)) * 10.0 ** g.uniform(-2, 2, n)
    B = g.standard_normal((3, n)) * 10.0 ** g.uniform(-3, 1.5, n)
    kin = 0.5 * rho * (v * v).sum(0) + 0.5 * (B * B).sum(0)
    p = kin * g.uniform(0, 2.0 ** -23, n) if cancel else 10.0 ** g.uniform(-4, 2, n)
    return rho, v, B, p, kin


@pytest.mark.gpu
@pytest.mark.parametrize("gamma", [1.4, 5.0 / 3.0, 2.0])
@pytest.mark.parametrize("flags", sorted(FLAGS))
def test_recovered_pressure(gpu, flags, gamma):
    L, n, ld = check_lib(flags), 1 << 18, np.longdouble
    for cancel in (False, True):
        rho, v, B, p, kin = states(n, 23, cancel)
        u = np.ascontiguousarray(np.stack([rho, *(rho * v), p / (gamma - 1) + kin, *B], 1), np.float32)
        got, fp64 = np.empty(n, np.float32), np.empty(n, np.float32)
        assert L.fp32_pressure(u.ctypes.data, n, gamma, got.ctypes.data, fp64.ctypes.data) == 0
        x, gm1 = u.astype(ld), ld(gamma) - 1
        half = ((x[:, 1] ** 2 + x[:, 2] ** 2 + x[:, 3] ** 2) / x[:, 0] + x[:, 5] ** 2 + x[:, 6] ** 2 + x[:, 7] ** 2) / 2
        exact, terms = gm1 * (x[:, 4] - half), gm1 * (x[:, 4] + half)
        ok = exact > 1e-9 + 2.0 ** -40 * terms      # above the floor, sign beyond doubt
        assert ok.mean() > 0.5
        err = np.abs(got.astype(ld) - exact)[ok]
        assert (err <= 2.0 ** -43 * terms[ok] + 0.501 * np.spacing(got[ok])).all()
        if cancel:
            old = np.abs(fp64.astype(ld) - exact)[ok]
            rms = [float(np.sqrt(((e / terms[ok]) ** 2).mean())) for e in (err, old)]
            assert rms[0] <= 1.02 * rms[1], rms
