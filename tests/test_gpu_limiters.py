"""Every slope limiter has code of its own in the face kernels: FP64 steps against
the oracle bit for bit, and a batch whose instances differ in their limiter
against single runs, in both precisions, in the split and the fused stage."""
import os

import numpy as np
import pytest

from oracle import pyoracle as P
from parity_util import oracle_kw


LIMITERS = ["1st", "noSL", "minmod", "VanLeer", "Superbee", "MC", "Koren", "Cada3rd"]


def config(gpu, limiter, precision):
    c = gpu.kh_config(3, precision)
    c.nroots_x = c.nroots_y = 3
    c.limiter = limiter.encode()
    return c


def simulation(gpu, configs, stage):
    os.environ["AMR2D_STAGE_KERNEL"] = stage
    try:
        return gpu.Simulation(configs).init()
    finally:
        del os.environ["AMR2D_STAGE_KERNEL"]


@pytest.mark.gpu
@pytest.mark.parametrize("stage", ["split", "fused"])
@pytest.mark.parametrize("limiter", LIMITERS)
def test_limiter_matches_the_oracle(gpu, limiter, stage):
    c = config(gpu, limiter, "fp64")
    sim, orc = simulation(gpu, c, stage), P.Oracle(**oracle_kw(c)).init()
    sim.run(3)
    orc.run(3)
    s, o = sim.state(), orc.state()
    assert np.array_equal(s["U"], o["U"]) and np.array_equal(s["Bi"], o["Bi"])


@pytest.mark.gpu
@pytest.mark.parametrize("stage", ["split", "fused"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_of_limiters(gpu, precision, stage):
    batch = simulation(gpu, [config(gpu, l, precision) for l in LIMITERS], stage)
    batch.run(3)
    for q, l in enumerate(LIMITERS):
        one = simulation(gpu, config(gpu, l, precision), stage)
        one.run(3)
        a, b = one.state(), batch.state(q)
        assert np.array_equal(a["U"], b["U"]) and np.array_equal(a["Bi"], b["Bi"]), l
