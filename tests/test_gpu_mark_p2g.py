"""The substep's fused marking and P2G (index order, no balls) against the
separate passes of the cell-ordered substep, at particle counts around its
runs of two and of four (ragged ends, both sides of the line between them),
power-of-two and other cell sizes, with particles that turn airborne."""
import numpy as np
import pytest

from fluid_solver import FluidSolver

pytestmark = pytest.mark.gpu

LINE = 3 << 19      # from this count on a thread takes four particles


@pytest.mark.parametrize("n,dx,count", [(24, 1.0, 1), (24, 1.0, 2), (24, 0.9, 5), (24, 1.0, 4099), (31, 0.9, 4098),
                                        (97, 1.0, LINE - 1), (97, 0.5, LINE), (97, 0.9, LINE + 3)])
def test_fused_marking_and_p2g(n, dx, count):
    out = []
    R, depth = 0.4 * n * dx, 0.12 * n * dx
    for order in (0, 1):
        fs = FluidSolver(nx=n, ny=n, nz=n, dx=dx, coreR=R - depth, terrainSeed=7, targetParticles=float(2 * count + 9000),
                         capacity=4 * count + 30000)
        fs.generateTerrain(7, R)
        fs.resetWater(depth)
        assert fs.scalars.nP >= count
        fs.set_nparticles(count)
        fs.set_params(pic=0.05, maxSpeed=3.0, thermalOn=0, sorTol=0.0, pressureIters=2, p2gCellOrder=order)
        fs.set_scalars(gRamp=1.5)
        r = np.random.default_rng(count)
        for k in ("pvx", "pvy", "pvz"):
            fs.upload(k, r.normal(scale=0.3, size=count).astype(np.float32))
        y = fs.download("py")[:count]
        high = r.random(count) < 0.02                    # into the sky, some of them into the topmost rows
        y[high] = r.uniform(0.8 * n * dx, n * dx, int(high.sum())).astype(np.float32)
        fs.upload("py", y)
        fs._substep(0.01)
        fs.synchronize()
        out.append({k: fs.download(k)[:(None if k == "cellType" else count)] for k in
                    ("cellType", "pflag", "px", "py", "pz", "pvx", "pvy", "pvz")})
        fs.close()
    a, b = out
    assert np.array_equal(a["cellType"], b["cellType"])
    assert np.array_equal(a["pflag"], b["pflag"])
    if count > 1000:
        assert np.any(a["pflag"] == 1) and np.any(a["pflag"] == 0) and np.any(a["cellType"] == 1)
    # face sums of a few tens of FP32 terms in another order (some 1e-6 of the
    # largest), two solve iterations and the FLIP difference on top: 2e-5;
    # positions follow by dt = 0.01 and their own rounding
    for k in ("pvx", "pvy", "pvz"):
        assert np.max(np.abs(a[k] - b[k])) <= 2e-5 * max(np.max(np.abs(b[k])), 1e-3), k
    for k in ("px", "py", "pz"):
        assert np.max(np.abs(a[k] - b[k])) <= 2 * np.spacing(np.float32(n * dx)) + 1e-6, k
