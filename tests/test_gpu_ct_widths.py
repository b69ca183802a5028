"""The CT kernels at each of their widths with four ghost layers, and the upwind
EMF at 224 and 128 threads per CTA: FP64 uniform meshes against the oracle bit
for bit, FP32 as a single mesh against the same mesh as one of several
instances (another width), bit for bit."""
import numpy as np
import pytest

from oracle import pyoracle as P
from parity_util import oracle_kw


def uniform(gpu, roots, precision, limiter, ct_type):
    c = gpu.ot_config(maxlevs=1, precision=precision, cfl=0.3, limiter=limiter)
    c.nroots_x = c.nroots_y = roots
    c.ct_type = ct_type
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("roots", [4, 18, 25])   # 416, 224 and 128 threads per CTA
@pytest.mark.parametrize("limiter,ct_type", [("WENO5", 1), ("WENO5", 2), ("MC", 2)])
def test_fp64_widths_match_the_oracle(gpu, limiter, ct_type, roots):
    c = uniform(gpu, roots, "fp64", limiter, ct_type)
    sim, orc = gpu.Simulation(c).init(), P.Oracle(**oracle_kw(c), lenx=c.lenx, leny=c.leny).init()
    for _ in range(4):   # the first steps have dt = 0
        sim.step()
        orc.step()
    a, b = sim.state(), orc.state()
    assert a["t"] == b["t"] > 0
    assert np.array_equal(a["U"], b["U"]) and np.array_equal(a["Bi"], b["Bi"])


@pytest.mark.gpu
@pytest.mark.parametrize("roots,copies", [(12, 4), (12, 7)])   # 144 leaves: 416 threads; 576: 224; 1008: 128
@pytest.mark.parametrize("limiter,ct_type", [("WENO5", 1), ("WENO5", 2), ("MC", 2)])
def test_fp32_mesh_does_not_depend_on_the_width(gpu, limiter, ct_type, roots, copies):
    c = uniform(gpu, roots, "fp32", limiter, ct_type)
    one, many = gpu.Simulation(c).init(), gpu.Simulation([c] * copies).init()
    one.run(4)
    many.run(4)
    a, b = one.state(), many.state(copies - 1)
    assert a["t"] == b["t"] > 0
    assert np.array_equal(a["U"], b["U"]) and np.array_equal(a["Bi"], b["Bi"])
