"""A NaN in a particle's position: every cell index derived from it is clamped
into the grid (a NaN converted from double to int is the most negative int,
not 0), the fluid marking latches the fault, the next synchronising call
returns WS_ERR_DEVICE, and the handle steps normally after a restore."""
import numpy as np
import pytest

from helpers import planet, to_device, PLAIN32
from fluid_solver import WsError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("field", ["px", "py", "pz"])
def test_nan_position_latched_and_recoverable(field, order):
    o = planet("planet32", **PLAIN32)
    o.set_scalars(gRamp=1.5)
    fs = to_device(o)
    fs.p2gCellOrder = order
    clean = fs.snapshot()
    bad = fs.download(field)
    bad[[0, 5, len(bad) - 1]] = np.nan
    fs.upload(field, bad)
    with pytest.raises(WsError) as ei:
        fs._substep(0.01)
        fs.synchronize()
    assert ei.value.code == -5 and "NaN" in str(ei.value)
    fs.restore(clean)
    fs._substep(0.01)
    fs.synchronize()
    assert np.all(np.isfinite(fs.download(field)))
    fs.close()
