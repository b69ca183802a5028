"""The FP32 path's pressure recovery with pairs of floats throughout, restated with
numpy on the CPU (cons2prim_cell<float> in amr2d_mhd_gb300/csrc/stage.cuh adds the
low parts of its sums without rounding, tests/test_gpu_fp32_pressure.py; here they
are rounded): its error against an exact rational evaluation, beside that of the
same sums taken in FP64 and rounded to FP32 at the end.  The unrounded pair has
to be good to 2^-43 of the subtracted terms (the bound of the form with FP64
sums), and the FP32 result within one and a half units of the rounded FP64
form's error."""
from fractions import Fraction

import numpy as np

from test_fp32_pressure import F, fma32, pressure_df, pressure_exact, sum_sq3, two_sum


def pressure_pairs(u, gh, gl):
    """(unrounded pair, FP32 result) of (gamma - 1)(E - (|m|^2/rho + |B|^2)/2)."""
    ir = F(F(1) / u[0])
    rl = F(fma32(-u[0], ir, F(1)) * ir)
    mh, ml = sum_sq3(u[1], u[2], u[3])
    bh, bl = sum_sq3(u[5], u[6], u[7])
    kh = F(mh * ir)
    kl = F(fma32(mh, ir, -kh) + F(F(mh * rl) + F(ml * ir)))
    sh, sl = two_sum(kh, bh)
    sl = F(sl + F(kl + bl))
    dh, dl = two_sum(u[4], F(F(-0.5) * sh))
    dl = fma32(F(-0.5), sl, dl)
    ph = F(gh * dh)
    pl = F(fma32(gh, dh, -ph) + fma32(gh, dl, F(gl * dh)))
    return Fraction(float(ph)) + Fraction(float(pl)), F(ph + pl)


def test_pair_recovery_error():
    rng = np.random.default_rng(17)
    for g in (1.4, 5.0 / 3.0, 2.0):
        gh = F(g - 1)
        gl = F((g - 1) - np.float64(gh))
        for n in range(1500):
            rho = 10.0 ** rng.uniform(-3, 3)
            v = rng.standard_normal(3) * 10.0 ** rng.uniform(-2, 2)     # up to Mach ~100
            B = rng.standard_normal(3) * 10.0 ** rng.uniform(-3, 1.5)
            p = 10.0 ** rng.uniform(-4, 2)
            u = np.array([rho, *(rho * v), 0.0, *B], dtype=F)
            ke = 0.5 * float(sum(float(x) ** 2 for x in u[1:4])) / float(u[0])
            me = 0.5 * float(sum(float(x) ** 2 for x in u[5:8]))
            u[4] = F(p / (g - 1) + ke + me)
            gm1, diff, scale = pressure_exact(u, g)
            exact = gm1 * diff
            pair, p32 = pressure_pairs(u, gh, gl)
            terms = float(gm1 * scale)
            assert abs(float(pair - exact)) / terms < 2.0 ** -43
            old = F(pressure_df(u, np.float64(g)))
            unit = float(np.spacing(abs(old))) if old else terms * 2.0 ** -43
            assert abs(float(Fraction(float(p32)) - exact)) <= abs(float(Fraction(float(old)) - exact)) + 1.5 * unit + \
                terms * 2.0 ** -43
