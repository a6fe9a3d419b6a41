"""The region solve (ws_sor_tb.cu) at the sizes where its plan can go wrong:
grids whose last bricks are partial, a grid with fewer bricks than CTAs, epochs
of two and of one iteration (odd counts, odd check cadence), oceans so deep that
the regions take the shorter halo or none fits, and a large grid. Its q is
bitwise that of the colour-list solves on the same system (ws_time_kernel id 7)
and, where the lists cover it, of one launch per colour (id 0)."""
import numpy as np
import pytest

from fluid_solver import FluidSolver

pytestmark = pytest.mark.gpu


def _planet(n, R, depth, particles):
    fs = FluidSolver(nx=n, ny=n, nz=n, dx=1.0, coreR=R - depth, terrainSeed=20260114,
                     targetParticles=float(particles), capacity=particles + 300000)
    fs.generateTerrain(20260114, R)
    fs.resetWater(depth)
    fs.set_params(pic=0.05, omega=1.7, maxSpeed=3.2, cfl=3.0, viscosity=5e-4, thermalOn=0, sorTol=0.0)
    fs.set_scalars(gRamp=1.5)
    return fs


# n, sea radius, depth, particles, iterations, paths the default solve may take
@pytest.mark.parametrize("n,R,depth,particles,iters,paths", [
    (12, 4.0, 2.5, 900, 5, (3,)),            # a handful of bricks: most CTAs own none
    (30, 11.5, 4.0, 9000, 1, (3,)),          # one iteration: an epoch of two half-sweeps only
    (45, 18.0, 6.0, 60000, 7, (3,)),         # partial bricks along each axis, odd count
    (101, 41.0, 9.0, 400000, 12, (3,)),
    (128, 56.0, 30.0, 1500000, 9, (3, 4)),   # thick ocean: shorter halo, or the in-launch fallback
    (172, 72.0, 10.0, 1200000, 11, (1,)),    # above 160^3
    (176, 80.0, 60.0, 2500000, 6, (1,)),     # above 160^3 and too thick: the lists
])
def test_region_solve_bitwise(n, R, depth, particles, iters, paths):
    fs = _planet(n, R, depth, particles)
    fs.pressureIters = iters
    fs._substep(0.01)                        # a warm q to start from
    for st in ("CLEAR_RASTER", "MARK_FLUID", "P2G"):
        fs.stage(st)
    fs.stage("FORCES", 0.01)
    q0 = fs.q.copy()
    q0[fs.cellType != 1] = 0.0
    fs.stage("PRESSURE")
    s = fs.scalars
    assert s.sorPath in paths and s.sorIters == iters
    q = fs.q.copy()
    assert np.all(np.isfinite(q)) and np.any(q != q0)
    fs.upload("q", q0)
    fs.time_kernel(7, 1)
    assert np.array_equal(q.view(np.uint32), fs.q.view(np.uint32))
    fs.upload("q", q0)
    fs.time_kernel(0, iters)
    assert np.array_equal(q.view(np.uint32), fs.q.view(np.uint32))
    fs.close()


@pytest.mark.parametrize("n,share,iters", [(64, 0.02, 60), (64, 0.2, 25), (96, 0.008, 80), (168, 0.01, 40)])
def test_scattered_fluid_bitwise(n, share, iters):
    """Scattered fluid cells: many bricks hold one or two, so a CTA often holds
    a neighbour's cell in its halo while its own lie beyond that neighbour's
    (each must still wait for the other before it overwrites an exchange
    buffer). 168^3 takes the large-grid route."""
    fs = FluidSolver(nx=n, ny=n, nz=n, dx=1.0, coreR=1.0, targetParticles=1000.0, capacity=1000)
    r = np.random.default_rng(n)
    ct = np.where(r.random((n, n, n)) < share, 1, 0).astype(np.uint8)
    for a in range(3):
        np.moveaxis(ct, a, 0)[[0, -1]] = 2
    fs.set_params(sorTol=0.0, pressureIters=iters, omega=1.7)
    fs.upload("cellType", ct.ravel())
    for k in ("u", "v", "w"):
        fs.upload(k, r.normal(size=fs.field_size(k)).astype(np.float32))
    q0 = np.where(ct.ravel() == 1, r.normal(size=n ** 3), 0).astype(np.float32)
    fs.upload("q", q0)
    for _ in range(3):                       # tags count on from solve to solve
        fs.upload("q", q0)
        fs.stage("PRESSURE")
    s = fs.scalars
    assert s.sorIters == iters
    q = fs.q.copy()
    assert np.all(np.isfinite(q)) and np.any(q != q0)
    fs.upload("q", q0)
    fs.time_kernel(0, iters)
    assert np.array_equal(q.view(np.uint32), fs.q.view(np.uint32))
    fs.close()


@pytest.mark.parametrize("check", [1, 3, 4, 10])
def test_check_cadence_stops_where_fixed_iterations_do(check):
    """Tolerance mode stops at a multiple of the cadence with the iterates of
    that many fixed iterations."""
    fs = _planet(45, 18.0, 6.0, 60000)
    fs.set_params(sorTol=1e-3, sorCheckEvery=check, sorMaxIters=400)
    for st in ("CLEAR_RASTER", "MARK_FLUID", "P2G"):
        fs.stage(st)
    fs.stage("FORCES", 0.01)
    q0 = fs.q.copy()
    q0[fs.cellType != 1] = 0.0
    fs.stage("PRESSURE")
    s = fs.scalars
    assert s.sorIters % check == 0 and 0 < s.sorIters < 400 and s.sorRelRes <= 1e-3
    q, rel = fs.q.copy(), s.sorRelRes
    assert abs(fs.residual() - rel) <= 1e-9 * rel
    fs.upload("q", q0)
    fs.set_params(sorTol=0.0, pressureIters=s.sorIters)
    fs.time_kernel(0, s.sorIters)
    assert np.array_equal(q.view(np.uint32), fs.q.view(np.uint32))
    fs.close()
