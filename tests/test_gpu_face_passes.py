"""The face passes over the active-brick list (four bricks per block, the last
group ragged, partial bricks along each axis) against the same substep with a
forced full pass, and a write of q alone, after which only the pressure setup
visits every brick: q ends at zero off the fluid, everything else as before."""
import numpy as np
import pytest

from fluid_solver import FluidSolver

pytestmark = pytest.mark.gpu
KEYS = ("u", "v", "w", "uO", "vO", "wO", "validU", "validV", "validW", "q", "cellType", "px", "pvx", "pvy", "pvz")


@pytest.mark.parametrize("dims,vorticity", [((13, 18, 21), 0.0), ((30, 31, 33), 0.0), ((32, 32, 32), 0.3), ((41, 38, 35), 0.0)])
def test_brick_passes_after_writes(dims, vorticity):
    n = min(dims)
    R, depth = 0.36 * n, 0.1 * n
    fs = FluidSolver(nx=dims[0], ny=dims[1], nz=dims[2], dx=1.0, coreR=R - depth, terrainSeed=3, targetParticles=9.0 * n * n,
                     capacity=400000)
    fs.generateTerrain(3, R)
    fs.resetWater(depth)
    fs.set_params(pic=0.05, maxSpeed=3.0, thermalOn=0, sorTol=0.0, pressureIters=6, vorticity=vorticity, viscosity=5e-4)
    fs.set_scalars(gRamp=1.5)
    for _ in range(3):
        fs._substep(0.01)
    snap = fs.snapshot()
    got = []
    for write in ("everything", "q", "q off the fluid"):
        fs.restore(snap)                                  # forces every brick once
        if write != "everything":
            # the same state reached again by an unforced substep: positions,
            # velocities and q are all that a substep takes over
            parts = {k: fs.download(k) for k in ("px", "py", "pz", "pvx", "pvy", "pvz", "pflag", "pcool", "q")}
            fs._substep(0.01)
            fs.synchronize()
            for k, a in parts.items():
                if k != "q":
                    fs.upload(k, a)
            q = parts["q"]
            if write == "q off the fluid":
                q = np.where(fs.download("cellType") == 1, q, np.float32(7.5)).astype(np.float32)
            fs.upload("q", q)
        fs.synchronize()
        fs._substep(0.01)
        fs.synchronize()
        got.append({k: fs.download(k) for k in KEYS})
        assert np.all(got[-1]["q"][got[-1]["cellType"] != 1] == 0)
    nP = fs.scalars.nP
    # a q left off the fluid may start a cell that fluid has just reached, so
    # that write is compared where it must agree: the types and valid flags
    a, b, c = got
    for k in KEYS:
        x, y = a[k], b[k]
        if k in ("px", "pvx", "pvy", "pvz"):
            x, y = x[:nP], y[:nP]
        if x.dtype == np.uint8:
            assert np.array_equal(x, y) and np.array_equal(x, c[k]), k
        else:
            # P2G's sums in another order, six iterations and the FLIP difference: 2e-5 of the largest
            assert np.max(np.abs(x - y)) <= 2e-5 * max(np.max(np.abs(x)), 1e-2), k
    fs.close()
