"""The CT face update keeps the reference's signs of zero (CT2D.cpp:78-92): where
the EMF is uniform, By loses -(1/dx) * (+0) = -0, so a By of -0 becomes +0, and
Bx loses +0, so a Bx of -0 stays."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("roots", [2, 20, 34])   # three widths of the CT kernels
def test_zero_faces_at_rest(gpu, roots, precision):
    c = gpu.kh_config(3, precision)
    c.nroots_x = c.nroots_y = roots
    sim = gpu.Simulation(c).init()
    U, Bi = sim.download("U"), sim.download("Bi")
    U[:] = 0.0
    U[:, 0], U[:, 4] = 1.0, 2.5
    Bi[:] = -0.0
    sim.upload("U", U)
    sim.upload("Bi", Bi)
    sim.run(1)
    B = sim.download("Bi")[:, :, 2:18, 2:18]
    assert (B == 0).all()
    assert np.signbit(B[:, 0]).all() and not np.signbit(B[:, 1]).any()
