"""Whole FP64 steps on states whose faces leave the Soft arithmetic's range
(components that are zero, subnormal or so small that their squares are), so
that the face kernels evaluate them again with the native operators: every
schedule of the face kernels against the oracle, bit for bit, and the adjoint's
face kernel against autograd."""
import os

import numpy as np
import pytest
import torch

import kh_reference as K
from oracle import pyoracle as P
from parity_util import oracle_kw
from test_gpu_adjoint import interior_only, kh_sim

SCHEDULES = [("split", "oneshot"), ("split", "persistent"), ("split", "dynamic"), ("fused", "oneshot"),
             ("fused", "dynamic")]
METHODS = [("MC", "RUSA", 2), ("MC", "HLLD", 2), ("VanLeer", "HLLE", 2), ("Koren", "HLLC", 2), ("WENO3", "HLLD", 2),
           ("WENO5", "RUSA", 4)]


def tiny(g, shape):
    """Values of order 1e-320 to 1e-2, and zeros of both signs."""
    return g.normal(0.0, 1.0, shape) * g.choice([0.0, 1e-320, 1e-310, 1e-200, 1e-160, 1e-155, 1e-20, 1e-2], shape)


@pytest.mark.gpu
@pytest.mark.parametrize("stage,face", SCHEDULES)
@pytest.mark.parametrize("limiter,flux,ng", METHODS)
def test_steps_match_the_oracle(gpu, limiter, flux, ng, stage, face):
    c = gpu.kh_config(3)
    c.nroots_x = c.nroots_y = 4
    c.limiter, c.flux, c.nghosts = limiter.encode(), flux.encode(), ng
    os.environ["AMR2D_STAGE_KERNEL"], os.environ["AMR2D_FACE_KERNEL"] = stage, face
    try:
        sim = gpu.Simulation(c).init()
    finally:
        del os.environ["AMR2D_STAGE_KERNEL"], os.environ["AMR2D_FACE_KERNEL"]
    orc = P.Oracle(**oracle_kw(c)).init()
    g = np.random.default_rng(41)
    U, Bi = sim.download("U"), sim.download("Bi")
    rho, v, b = g.uniform(1.0, 1.1, U[:, 0].shape), tiny(g, U[:, 1:4].shape), tiny(g, U[:, 5:8].shape)
    U[:, 0], U[:, 1:4], U[:, 5:8] = rho, rho[:, None] * v, b
    U[:, 4] = g.uniform(1.0, 1.1, rho.shape) / (5.0 / 3.0 - 1)
    Bi[:] = tiny(g, Bi.shape)
    for f, a in (("U", U), ("Bi", Bi)):
        sim.upload(f, a)
        orc.set(f, a)
    for _ in range(2):
        sim.step()
        orc.step()
    s, o = sim.state(), orc.state()
    assert np.isfinite(o["U"]).all()
    assert np.array_equal(s["U"], o["U"]) and np.array_equal(s["Bi"], o["Bi"])


@pytest.mark.gpu
def test_adjoint_of_such_a_state(gpu):
    n, h = 256, 1.0 / 256
    sim, c = kh_sim(gpu)
    sim.run(3)
    ic = sim.tree()[1]
    g = np.random.default_rng(43)
    U = K.from_blocks(sim.download("U"), ic)
    U[3], U[7] = tiny(g, U[3].shape), tiny(g, U[7].shape)
    sim.upload("U", K.to_blocks(U, ic))
    B0 = K.from_blocks(sim.download("Bi"), ic)
    lU = g.standard_normal((8, n, n))
    sim.adjoint_enable(True)
    sim.step()
    sim.adjoint_seed("U", interior_only(K.to_blocks(lU, ic)))
    sim.adjoint_step()
    gU = K.from_blocks(sim.adjoint_read("U"), ic)
    U0 = torch.from_numpy(U.copy()).requires_grad_(True)
    U1, _, _ = K.step(U0, torch.from_numpy(B0[0].copy()), torch.from_numpy(B0[1].copy()), c.dt_fixed, c.gamma, h)
    (torch.from_numpy(lU) * U1).sum().backward()
    for k in (0, 1, 2, 4, 5, 6):
        ref = U0.grad[k].numpy()
        assert np.abs(gU[k] - ref).max() < 1e-10 * np.abs(ref).max(), k
    assert np.isfinite(gU).all()
