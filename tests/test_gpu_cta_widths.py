"""The per-leaf kernels choose their CTA width by the number of leaves (wide
CTAs for few leaves).  Uniform meshes on both sides of every line: FP64 against
the oracle bit for bit (state and, through t, the CFL reduction), FP32 as a
single mesh against the same mesh as one of several instances of a handle, bit
for bit."""
import numpy as np
import pytest

from oracle import pyoracle as P
from parity_util import oracle_kw


def uniform(gpu, roots, precision):
    c = gpu.ot_config(maxlevs=1, precision=precision, cfl=0.3, limiter="MC")
    c.nroots_x = c.nroots_y = roots
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("roots", [4, 16, 18, 20, 26, 36])
def test_fp64_meshes_match_the_oracle(gpu, roots):
    c = uniform(gpu, roots, "fp64")
    sim, orc = gpu.Simulation(c).init(), P.Oracle(**oracle_kw(c), lenx=c.lenx, leny=c.leny).init()
    for _ in range(4):   # the first steps have dt = 0
        sim.step()
        orc.step()
    a, b = sim.state(), orc.state()
    assert a["t"] == b["t"] > 0
    assert np.array_equal(a["U"], b["U"]) and np.array_equal(a["Bi"], b["Bi"])


@pytest.mark.gpu
@pytest.mark.parametrize("roots,copies", [(16, 2), (16, 4), (17, 8), (4, 70)])
def test_fp32_mesh_does_not_depend_on_the_other_instances(gpu, roots, copies):
    c = uniform(gpu, roots, "fp32")
    one, many = gpu.Simulation(c).init(), gpu.Simulation([c] * copies).init()
    one.run(4)
    many.run(4)
    for q in (0, copies - 1):
        a, b = one.state(), many.state(q)
        assert a["t"] == b["t"] > 0
        assert np.array_equal(a["U"], b["U"]) and np.array_equal(a["Bi"], b["Bi"])
