"""The FP32 path stops with AMR_E_NAN (or HLLC's own code) on a face state of
negative pressure or density wherever the FP64 path does, whose fast speed
(misc.cpp:71-79) takes their square roots: Cada's limiter, third order and
unlimited where the jumps are below the cell size, drives the left pressure
(density) of a face beside a small drop below zero.  (HLLE and, for the
pressure, HLLD take minima and maxima that pass over a NaN on one side.)"""
import numpy as np
import pytest

AMR_E_NAN, AMR_E_HLLC = -6, -8


def sim_of(gpu, flux, precision, split):
    import os
    c = gpu.kh_config(3, precision)
    c.nroots_x = c.nroots_y = 2
    c.limiter, c.flux = b"Cada3rd", flux.encode()
    os.environ["AMR2D_STAGE_KERNEL"] = "split" if split else "fused"
    try:
        return gpu.Simulation(c).init()
    finally:
        del os.environ["AMR2D_STAGE_KERNEL"]


def state(sim, drop):
    """At rest but for a uniform field; a drop of `drop` across x = 1/2 and back."""
    U, Bi = sim.download("U"), sim.download("Bi")
    x0 = np.array([ic[0] for ic in sim.tree()[1]])
    i = np.arange(20) - 2
    x = (x0[:, None] + i) % 32                              # cell column of each block's columns
    low = ((x >= 8) & (x < 24))[:, None, :] * np.ones((1, 20, 1))
    rho, p = np.ones_like(low), np.ones_like(low)
    if drop == "pressure":
        p = np.where(low, 0.003, 0.03)
    elif drop == "density":
        rho = np.where(low, 0.003, 0.03)
    b = (0.3, 0.4, 0.2)
    U[:] = 0.0
    U[:, 0], U[:, 5], U[:, 6], U[:, 7] = rho, *b
    U[:, 4] = p / (5.0 / 3.0 - 1) + 0.5 * (b[0] ** 2 + b[1] ** 2 + b[2] ** 2)
    Bi[:, 0], Bi[:, 1] = b[0], b[1]
    return U, Bi


@pytest.mark.gpu
@pytest.mark.parametrize("split", [False, True], ids=["fused", "split"])
@pytest.mark.parametrize("flux", ["RUSA", "HLLE", "HLLC", "HLLD"])
@pytest.mark.parametrize("drop", ["pressure", "density", "none"])
def test_negative_face_state_is_trapped(gpu, drop, flux, split):
    def outcome(precision):
        sim = sim_of(gpu, flux, precision, split)
        U, Bi = state(sim, drop)
        sim.upload("U", U)
        sim.upload("Bi", Bi)
        try:
            sim.run(1)
        except gpu.AmrError as e:
            return e.code
        return 0
    want = outcome("fp64")
    if drop == "none":
        assert want == 0
    elif flux in ("RUSA", "HLLC"):
        assert want in (AMR_E_NAN, AMR_E_HLLC)
    assert outcome("fp32") == want
