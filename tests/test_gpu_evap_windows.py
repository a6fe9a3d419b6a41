"""Evaporation where the blocks of the outcome table are shared out over the
windows that hold candidates: a planet of one window (fewer candidates than 4096,
a single ragged one) and one of many, in a store of particles whose count gives
several times as many possible windows. Ejections, flags and the final stream
state against the oracle's serial walk."""
import math

import numpy as np
import pytest

from helpers import planet, to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,windows", [("planet32", 1), ("planet128", 20)])
def test_shared_windows(name, windows):
    o = planet(name, pic=0.05, omega=1.7, maxSpeed=3.2, cfl=3.0, pressureIters=20, thermalOn=1, sunActivity=2.0,
               evapIntensity=1.0)
    c = o.nx / 2
    o.set(sunPos=[c + 3 * o.scalars.oceanR * math.cos(0.4), c + 3 * o.scalars.oceanR * math.sin(0.4), c])
    o.set_scalars(gRamp=1.5)
    o.substep(0.01)
    o.stage("splat_density")
    nP = o.nP
    o.pT[:nP] = np.random.default_rng(3).uniform(0.2, 1.0, nP).astype(np.float32)
    fs = to_device(o, with_grid=True)
    o.stage("update_evaporation", 1 / 12)
    fs.stage("EVAPORATION", 1 / 12)
    so, sg = o.scalars, fs.scalars
    assert so.evapCount > 0 and sg.evapCount == so.evapCount
    assert sg.evS == so.evS
    assert np.array_equal(fs.pflag, o.pflag[:nP])
    # an ejection takes 6 draws beside the candidate's own, so the stream tells the candidates' number
    draws, s = 0, 0x51ab3c77
    while s != so.evS:
        s = (s * 1664525 + 1013904223) % 2 ** 32
        draws += 1
    assert (draws - 6 * so.evapCount + 4095) // 4096 >= windows
    fs.close()
