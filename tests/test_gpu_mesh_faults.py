"""A mesh call that answers with a latched fault leaves the last mesh (and the
metaball field) as they were: vertices, count and lattice."""
import ctypes as C

import numpy as np
import pytest

from helpers import planet, to_device, PLAIN32
from fluid_solver import WsError

pytestmark = pytest.mark.gpu


def _mesh(fs, kind):
    """The mesh that the handle shows: positions, normals, count."""
    n = C.c_int64()
    p, q = C.c_void_p(), C.c_void_p()
    fs._check(getattr(fs._L, "ws_%s_device" % kind)(fs._h, C.byref(p), C.byref(q), C.byref(n)))
    pos, nrm = (np.zeros((n.value, 3), np.float32) for _ in range(2))
    fs._check(getattr(fs._L, "ws_%s_download" % kind)(fs._h, pos.ctypes.data, nrm.ctypes.data, n.value))
    return n.value, pos, nrm


def _build(fs, kind, arg):
    n, vol = C.c_int64(), C.c_double()
    if kind == "surface":
        fs._check(fs._L.ws_surface_mesh(fs._h, arg, C.byref(n), C.byref(vol)))
    else:
        fs._check(fs._L.ws_metaball_mesh(fs._h, 0.5, arg, C.byref(n), C.byref(vol)))


def _field(fs):
    m = C.c_int32()
    fs._check(fs._L.ws_metaball_field(fs._h, None, 0, C.byref(m)))
    f = np.zeros((m.value + 1) ** 3 if m.value else 0, np.float32)
    if len(f):
        fs._check(fs._L.ws_metaball_field(fs._h, f.ctypes.data, len(f), C.byref(m)))
    return m.value, f


# the lattice of the failing metaball call: the same, a smaller and a larger one
@pytest.mark.parametrize("kind,arg", [("surface", None), ("metaball", 1.0), ("metaball", 0.6), ("metaball", 1.6)])
@pytest.mark.parametrize("first", [True, False])
def test_latched_fault_leaves_the_mesh(kind, arg, first):
    o = planet("planet32", **PLAIN32)
    o.set_scalars(gRamp=1.5)
    fs = to_device(o)
    fs.stage("SPLAT")
    iso = 1.0
    if not first:
        _build(fs, kind, iso if kind == "surface" else 1.0)
        assert _mesh(fs, kind)[0] > 1000
    old, field = _mesh(fs, kind), _field(fs)
    fs.upload("dens", 3 * fs.download("dens"))       # another surface and other particles
    px = fs.download("px") + np.float32(0.4)
    px[3] = np.nan
    fs.upload("px", px)
    fs._substep(0.01)
    with pytest.raises(WsError) as ei:
        _build(fs, kind, iso if kind == "surface" else arg)
    assert ei.value.code == -5
    now = _mesh(fs, kind)
    assert now[0] == old[0]
    for a, b in zip(old[1:], now[1:]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    m, f = _field(fs)
    assert m == field[0] and np.array_equal(f.view(np.uint32), field[1].view(np.uint32))
    fs.close()


def test_metaball_lattice_limit():
    """A long thin grid asks for an nx^3 lattice: beyond 32-bit corner indices
    (1625^3 < 2^32 < 1626^3 corners) the call is refused."""
    from fluid_solver import FluidSolver
    assert 1625 ** 3 < 2 ** 32 < 1626 ** 3
    fs = FluidSolver(nx=1700, ny=4, nz=4, dx=1.0, coreR=1.0, targetParticles=10.0, capacity=100)
    fs.set_scalars(spacing=0.5, nP=0)
    for detail in (1.0, 1.6, 0.9558):                     # 0.9558 * 1700 = 1624.9, rounded to 1625
        with pytest.raises(WsError) as ei:
            _build(fs, "metaball", detail)
        assert ei.value.code == -7
    assert _mesh(fs, "metaball")[0] == 0
    fs.close()
