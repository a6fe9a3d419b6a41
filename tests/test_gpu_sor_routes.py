"""Which solve runs, told by ws_timed_solve on every grid size and by sorPath
where that has a number of its own, and the routes that no ordinary planet takes:
systems too thick for the regions, fluid on the outermost layer, and the
grid-wide lists with several cells a thread. Every q is bitwise that of one launch
per colour (ws_time_kernel id 0)."""
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


def _system(n, share, iters, shell, **params):
    """Fluid in `share` of the cells, the outermost layer closed (shell) or as wet as the rest."""
    fs = FluidSolver(nx=n, ny=n, nz=n, dx=1.0, coreR=1.0, targetParticles=1000.0, capacity=1000)
    r = np.random.default_rng(n)
    ct = np.where(r.random((n, n, n)) < share, 1, 0).astype(np.uint8)
    if shell:
        for a in range(3):
            np.moveaxis(ct, a, 0)[[0, -1]] = 2
    fs.set_params(**dict(dict(sorTol=0.0, pressureIters=iters, omega=1.7), **params))
    fs.upload("cellType", ct.ravel())
    for k in ("u", "v", "w"):
        fs.upload(k, r.normal(size=fs.field_size(k)).astype(np.float32))
    q0 = np.where(ct.ravel() == 1, r.normal(size=n ** 3), 0).astype(np.float32)
    fs.upload("q", q0)
    fs.stage("PRESSURE")
    return fs, q0, fs.q.copy()


def _bitwise(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


def _colours(fs, q0, iters):
    fs.upload("q", q0)
    fs.time_kernel(0, iters)
    return fs.q.copy()


# n, sea radius, depth, particles: the default solve's route, and that of the list solve on the same system
@pytest.mark.parametrize("n,R,depth,particles,route,lists", [
    (30, 11.5, 4.0, 9000, 3, 2),
    (128, 52.0, 8.0, 1800000, 3, 2),         # 52k cells a colour: 16 CTAs of a cluster hold them
    (172, 72.0, 10.0, 1200000, 3, 1),        # above 160^3, thin: regions
    (176, 80.0, 60.0, 2500000, 3, 1),        # thick: regions with the shorter halo
])
def test_route(n, R, depth, particles, route, lists):
    fs = _planet(n, R, depth, particles)
    fs.pressureIters = 6
    fs._substep(0.01)
    q0 = fs.q.copy()
    want = _colours(fs, q0, 6)
    for kernel, path in ((6, route), (7, lists)):
        fs.upload("q", q0)
        fs.time_kernel(kernel, 1)
        got = fs.timed_solve()
        assert got[:2] == (path, 6) and got[2] > 0
        assert _bitwise(fs.q.copy(), want)
    fs.close()


def test_lists_with_several_cells_a_thread():
    """The grid-wide list solve of a 256^3 planet (about 680k fluid cells): contiguous
    ranges of each colour list per CTA and waits for neighbouring ranges only."""
    fs = _planet(256, 110.0, 12.0, 4000000)
    fs.pressureIters = 24
    fs._substep(0.01)
    q0 = fs.q.copy()
    assert fs.scalars.nFluid > 2 * 148 * 1024
    fs.time_kernel(7, 1)
    assert fs.timed_solve()[:2] == (1, 24)
    got = fs.q.copy()
    assert _bitwise(got, _colours(fs, q0, 24))
    fs.upload("q", q0)
    fs.time_kernel(6, 1)                     # the default on this grid: regions
    assert fs.timed_solve()[:2] == (3, 24)
    assert _bitwise(fs.q.copy(), got)
    fs.close()


@pytest.mark.parametrize("iters", [1, 6])
def test_owned_bricks_in_global_memory(iters):
    """A 128^3 grid nine tenths full: 12,700 cells a CTA with their halos do not fit."""
    fs, q0, q = _system(128, 0.9, iters, True)
    assert fs.scalars.sorPath == 4 and fs.scalars.sorIters == iters
    assert _bitwise(q, _colours(fs, q0, iters)) and not _bitwise(q, q0)
    fs.close()


def test_lists_after_regions_that_do_not_fit():
    """The same system above 160^3: the region launch leaves it to the list kernels behind it."""
    fs, q0, q = _system(168, 0.9, 5, True)
    assert fs.scalars.sorPath == 1 and fs.scalars.sorIters == 5
    assert _bitwise(q, _colours(fs, q0, 5)) and not _bitwise(q, q0)
    fs.upload("q", q0)
    fs.time_kernel(6, 1)
    assert fs.timed_solve()[:2] == (1, 5)
    assert _bitwise(fs.q.copy(), q)
    fs.close()


def test_owned_bricks_stop_where_the_regions_would():
    """Tolerance mode of that route: stops at a check, with the iterates of as many fixed iterations."""
    fs, q0, q = _system(128, 0.9, 0, True, sorTol=0.3, sorCheckEvery=3, sorMaxIters=60)
    s = fs.scalars
    assert s.sorPath == 4 and s.sorIters % 3 == 0 and 0 < s.sorIters < 60 and s.sorRelRes <= 0.3
    assert abs(fs.residual() - s.sorRelRes) <= 1e-9 * s.sorRelRes
    assert _bitwise(q, _colours(fs, q0, s.sorIters))
    fs.close()


@pytest.mark.parametrize("n,path,timed", [(20, 4, 4), (33, 4, 4), (164, 1, 1)])
def test_fluid_on_the_outermost_layer(n, path, timed):
    """Fluid on the outermost layer (only a caller's upload brings it) is never swept but
    its pressure is read, which the regions do not hold."""
    fs, q0, q = _system(n, 0.3, 5, False)
    assert fs.scalars.sorPath == path and fs.scalars.sorIters == 5
    assert _bitwise(q, _colours(fs, q0, 5)) and not _bitwise(q, q0)
    fs.upload("q", q0)
    fs.time_kernel(6, 1)
    assert fs.timed_solve()[:2] == (timed, 5)
    assert _bitwise(fs.q.copy(), q)
    fs.upload("q", q0)
    fs.time_kernel(7, 1)                     # the lists: grid-wide, though a cluster would hold the small ones
    assert fs.timed_solve()[:2] == (1, 5)
    assert _bitwise(fs.q.copy(), q)
    fs.close()


def test_route_after_the_outermost_layer_has_dried():
    """The next cell types, with a closed layer and no raster pass between, take the regions again."""
    fs, q0, _ = _system(33, 0.3, 5, False)
    assert fs.scalars.sorPath == 4
    ct = fs.cellType.reshape(33, 33, 33).copy()
    for a in range(3):
        np.moveaxis(ct, a, 0)[[0, -1]] = 2
    fs.upload("cellType", ct.ravel())
    q0 = np.where(ct.ravel() == 1, q0, 0).astype(np.float32)
    fs.upload("q", q0)
    fs.stage("PRESSURE")
    assert fs.scalars.sorPath == 3
    q = fs.q.copy()
    assert _bitwise(q, _colours(fs, q0, 5))
    fs.close()


def test_grid_longer_than_the_region_plan():
    """Brick coordinates of the plan hold 8 bits: beyond 1020 cells an axis the lists solve, in one cluster."""
    shape = (9, 10, 1032)
    fs = FluidSolver(nx=shape[2], ny=shape[1], nz=shape[0], dx=1.0, coreR=1.0, targetParticles=1000.0, capacity=1000)
    r = np.random.default_rng(5)
    ct = np.where(r.random(shape) < 0.4, 1, 0).astype(np.uint8)
    for a in range(3):
        np.moveaxis(ct, a, 0)[[0, -1]] = 2
    fs.set_params(sorTol=0.0, pressureIters=7, omega=1.7)
    fs.upload("cellType", ct.ravel())
    for k in ("u", "v", "w"):
        fs.upload(k, r.normal(size=fs.field_size(k)).astype(np.float32))
    q0 = np.where(ct.ravel() == 1, r.normal(size=ct.size), 0).astype(np.float32)
    fs.upload("q", q0)
    fs.stage("PRESSURE")
    assert fs.scalars.sorPath == 2 and fs.scalars.sorIters == 7
    q = fs.q.copy()
    assert _bitwise(q, _colours(fs, q0, 7)) and not _bitwise(q, q0)
    fs.close()
