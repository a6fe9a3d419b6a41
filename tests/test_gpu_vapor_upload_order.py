"""Two uploads in a row, the second bringing the first vapour flags: the
temperature of the first was left on its way beside the substeps, and the
second's temperature, or the vapour pass of the next substep where it brings
none, comes after it."""
import numpy as np
import pytest
import torch

from fluid_solver import FluidSolver

pytestmark = pytest.mark.gpu
N = 3_000_000                                    # 12 MB of temperatures, far more than the planet's particles


def _pinned(a):
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    v = t.numpy().view(a.dtype)
    v[:] = a
    return v


@pytest.mark.parametrize("second", ["flags and temperature", "flags only"])
def test_first_vapour_after_a_pending_temperature(second):
    names = ("px", "py", "pz", "pvx", "pvy", "pvz", "pT", "pAir", "pflag")
    out, base = {}, None
    for how in ("fields", "state"):
        fs = FluidSolver(nx=32, ny=32, nz=32, dx=1.0, coreR=9.0, terrainSeed=1, targetParticles=9000.0, capacity=N)
        fs.generateTerrain(1, 12.0)
        fs.resetWater(3.0)
        n = fs.scalars.nP
        if base is None:
            base = {k: fs.download(k, N).copy() for k in names}
            vap = np.zeros(N, bool)
            vap[:n:7] = True
            base["pAir"][vap] = 1.0
            old = np.full(N, 0.35, np.float32)
            new = np.where(np.arange(N) % 14 == 0, 0.05, 0.35).astype(np.float32)    # half of the parcels rain out
            flags = np.where(vap, 2, 0).astype(np.uint8)
            first_T, last_T = (old, new) if second == "flags and temperature" else (new, new)
        one = dict(base, pT=first_T, pflag=np.zeros(N, np.uint8))
        two = {"pflag": flags}
        if second == "flags and temperature":
            two["pT"] = last_T
        fs.set_scalars(cfS=1, bfS=2)
        if how == "state":                       # nothing between the calls joins the copies
            kept = [{k: _pinned(v) for k, v in part.items()} for part in (one, two)]
            fs.upload_state(kept[0], N)
            fs.upload_state(kept[1], N)
        else:
            for k, v in [*one.items(), *two.items()]:
                fs.upload(k, v)
        fs._substep(0.01)
        fs.synchronize()
        out[how] = {k: fs.download(k, N) for k in ("px", "py", "pz", "pT", "pflag")}
        fs.close()
    for how in out:
        assert np.array_equal(out[how]["pT"], last_T), how
        assert np.count_nonzero(out[how]["pflag"] == 4) > 0, how
    assert np.array_equal(out["state"]["pflag"][vap], out["fields"]["pflag"][vap])
    for k in ("px", "py", "pz"):
        assert np.allclose(out["state"][k][vap], out["fields"][k][vap], rtol=0, atol=1e-4), k

