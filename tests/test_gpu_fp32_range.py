"""The FP32 path at the ends of the float range, where MUFU's reciprocal
flushes: a contact at rest (uniform pressure and field, no velocity) whose
densities lie above 2^126, so that every 1/rho of the face solver is below the
smallest normal float.  Rusanov's dissipation spreads the contact by
sqrt(gamma p / rho) / 2 per unit of time; compared with the FP64 path.  The
tolerance: the relative error of a speed is below 20 units of 2^-23 and moves
less than half of the density in the three steps."""
import os

import numpy as np
import pytest


def run(gpu, precision, split, limiter):
    c = gpu.kh_config(3, precision)
    c.nroots_x = c.nroots_y = 2
    c.limiter, c.dt_fixed, c.t_end = limiter.encode(), 0.05, 10.0
    os.environ["AMR2D_STAGE_KERNEL"] = "split" if split else "fused"
    try:
        sim = gpu.Simulation(c).init()
    finally:
        del os.environ["AMR2D_STAGE_KERNEL"]
    U, Bi = sim.download("U"), sim.download("Bi")
    x = (np.array([ic[0] for ic in sim.tree()[1]])[:, None] + np.arange(20) - 2) % 32
    rho = np.where((x >= 8) & (x < 24), 0.95e38, 1.55e38)[:, None, :] * np.ones((1, 20, 1))
    U[:] = 0.0
    U[:, 0], U[:, 5], U[:, 6] = rho, 1e17, 2e17
    U[:, 4] = 1e36 / (5.0 / 3.0 - 1) + 0.5 * (1e34 + 4e34)
    Bi[:, 0], Bi[:, 1] = 1e17, 2e17
    sim.upload("U", U)
    sim.upload("Bi", Bi)
    sim.run(3)
    return U[:, 0, 2:18, 2:18], sim.download("U")[:, 0, 2:18, 2:18]


@pytest.mark.gpu
@pytest.mark.parametrize("limiter", ["1st", "minmod", "MC"])
@pytest.mark.parametrize("split", [False, True], ids=["fused", "split"])
def test_contact_of_densities_above_2_126(gpu, split, limiter):
    before, want = run(gpu, "fp64", split, limiter)
    got = run(gpu, "fp32", split, limiter)[1]
    assert (np.abs(want - before) / before).max() > 0.01      # the contact has spread
    assert (np.abs(got - want) / want).max() < 20 * 2.0 ** -23
