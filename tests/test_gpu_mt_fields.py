"""The marching-tets passes on corner fields that exercise every sign pattern,
against the oracle's build on the same field, bit for bit and in order: noise
around iso, corners exactly at iso, NaN corners, lattices around the passes'
blocks (1024 cells, 16 listed cells), axes of different lengths, a cell size
that is no power of two, and a mesh that outgrows the vertex buffers."""
import numpy as np
import pytest

from fluid_solver import FluidSolver
from oracle.oracle import mt_mesh_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,dx,kind", [((8, 9, 10), 1.0, "noise"), ((8, 8, 16), 1.0, "steps"), ((8, 9, 41), 0.7, "noise"),
                                          ((10, 11, 13), 0.5, "steps"), ((24, 25, 26), 1.0, "noise"), ((16, 16, 16), 0.9, "nan"),
                                          ((33, 31, 20), 1.0, "smooth")])
def test_fields(dims, dx, kind):
    nx, ny, nz = dims
    fs = FluidSolver(nx=nx, ny=ny, nz=nz, dx=dx, coreR=1.0, targetParticles=100.0, capacity=1000)
    r = np.random.default_rng(nx * ny + nz)
    shape = (nz + 1, ny + 1, nx + 1)
    for rounds in range(3):                              # the second mesh is larger, the third as large
        if kind == "smooth":
            z, y, x = np.meshgrid(*[np.linspace(0, 3 + rounds, s) for s in shape], indexing="ij")
            f = 1 + np.sin(2 * x) * np.cos(3 * y) + 0.5 * np.sin(z + x)
        else:
            f = 1 + r.normal(size=shape) * (1.0 if rounds else 0.2) - (0.0 if rounds else 0.5)
        if kind == "steps":
            f = np.round(f * 2) / 2                      # many corners exactly at iso
        f = f.astype(np.float32)
        if kind == "nan":
            f[r.random(shape) < 0.01] = np.nan
        fs.upload("dens", f.ravel())
        vol, pos, nrm = fs.surface_mesh(1.0)
        vref, pref, nref = mt_mesh_field(f.ravel(), nx, ny, nz, dx, 1.0)
        assert len(pos) == len(pref) and (rounds == 0 or len(pref) > 0)   # a first steps field may stay below iso
        assert np.array_equal(pos, pref, equal_nan=True) and np.array_equal(nrm, nref, equal_nan=True)
        v2, n2 = fs.mt_volume(1.0)
        assert n2 == len(pref)
        if kind != "nan":
            # sums of at most 2e5 triangles whose terms reach size^3, in another order
            assert abs(vol - abs(vref)) <= 1e-12 * abs(vref) + 1e-11 * (nx * ny * nz * dx ** 3)
            assert vol == v2
    fs.close()
