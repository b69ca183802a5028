"""Every line of the autotuner's report is a launch of its own: no description
twice, and the one-shot face kernel at the widths it runs at (32 and 128)."""
import re

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_report_names_what_ran(gpu, precision):
    sim = gpu.Simulation(ic="rotor", limiter="MC", flux="HLLD", cfl=0.4, maxlevs=3, precision=precision).init()
    sim.run(5)
    names = [re.sub(r"^[* ] |: .*", "", l) for l in sim.autotune(1).strip().splitlines()]
    assert len(set(names)) == len(names) == 42
    oneshot = {int(m.group(1)) for m in (re.match(r"split faces (\d+) cells", n) for n in names) if m}
    assert oneshot == {32, 128}
    assert not any(n.startswith("fused") and "faces" in n for n in names)   # it has no face kernel
