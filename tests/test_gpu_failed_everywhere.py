"""A step that fails in every cell and face: it reports a failure as any other,
the engine stays stopped, and the step takes a few steps' time (the claims of
the error record stay on the device)."""
import time

import numpy as np
import pytest


@pytest.mark.gpu
def test_nan_in_every_cell(gpu):
    c = gpu.kh_config(3, "fp64")
    c.nroots_x = c.nroots_y = 48
    sim = gpu.Simulation(c).init()
    sim.run(3)
    t = time.perf_counter()
    sim.run(5)
    good = (time.perf_counter() - t) / 5
    U = sim.download("U")
    U[:, 4] = np.nan
    sim.upload("U", U)
    t = time.perf_counter()
    with pytest.raises(gpu.AmrError) as e:
        sim.run(1)
    bad = time.perf_counter() - t
    assert e.value.code == -6 and "device check failed (code 2)" in str(e.value)
    with pytest.raises(gpu.AmrError):
        sim.run(1)
    assert bad < 15 * good, (bad, good)
