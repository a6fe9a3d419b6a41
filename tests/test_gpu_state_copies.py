"""State uploads and downloads: pinned buffers small enough for the copying
kernel, the same buffers off 16-byte alignment, pageable ones, counts with a
ragged tail and on both sides of the 4 MB line all move the same bytes, and
vapour flags brought by an upload are seen by the next substep."""
import numpy as np
import pytest
import torch

from fluid_solver import FluidSolver

pytestmark = pytest.mark.gpu
FIELDS = {"px": np.float32, "py": np.float32, "pz": np.float32, "pvx": np.float32, "pvy": np.float32, "pvz": np.float32,
          "pT": np.float32, "pflag": np.uint8, "pcool": np.uint8, "pDepth": np.uint8}


def _pinned(n, dt, off):
    t = torch.empty(n * dt().itemsize + 64, dtype=torch.uint8, pin_memory=True)
    return t.numpy()[off:off + n * dt().itemsize].view(dt)


@pytest.mark.parametrize("kind", ["pinned", "offset", "pageable", "mixed"])
@pytest.mark.parametrize("count", [1, 5, 4097, 150001])     # 31 bytes a particle: the last lies beyond 4 MB
def test_round_trip(kind, count):
    fs = FluidSolver(nx=24, ny=24, nz=24, dx=1.0, coreR=6.0, targetParticles=1000.0, capacity=160000)
    fs.set_nparticles(count)
    r = np.random.default_rng(count)
    src, dst = {}, {}
    for i, (k, dt) in enumerate(FIELDS.items()):
        how = ("pinned", "offset", "pageable")[i % 3] if kind == "mixed" else kind
        for d in (src, dst):
            d[k] = np.empty(count, dt) if how == "pageable" else _pinned(count, dt, 4 if how == "offset" else 0)
        src[k][:] = r.integers(0, 2, count) if dt is np.uint8 else r.normal(size=count)
        dst[k][:] = 7
    for again in range(2):                                  # the second upload reads rewritten buffers
        if again:
            for k in FIELDS:
                src[k][:] = src[k][::-1].copy()
        fs.upload_state(src, count)
        fs.download_state(dst, count)
        for k in FIELDS:
            assert np.array_equal(dst[k].view(np.uint8), src[k].view(np.uint8)), k
            assert np.array_equal(fs.download(k, count).view(np.uint8), src[k].view(np.uint8)), k
    fs.close()


def test_vapour_seen_after_pinned_upload():
    names = ("px", "py", "pz", "pvx", "pvy", "pvz", "pT", "pflag")
    out, first = {}, None
    for how in ("fields", "state"):                         # a handle each: the flag stays once seen
        fs = FluidSolver(nx=32, ny=32, nz=32, dx=1.0, coreR=9.0, terrainSeed=1, targetParticles=9000.0, capacity=30000)
        fs.generateTerrain(1, 12.0)
        fs.resetWater(3.0)
        n = fs.scalars.nP
        if first is None:
            first = {k: fs.download(k, n).copy() for k in names}
            first["pflag"][::50] = 2
            first["pT"][::50] = 0.4
        state = {k: _pinned(n, FIELDS[k], 0) for k in names}
        for k in names:
            state[k][:] = first[k]
        if how == "fields":
            for k in names:
                fs.upload(k, first[k])
        else:
            fs.upload_state(state, n)
        fs.set_scalars(cfS=1, bfS=2)
        fs._substep(0.01)
        fs.synchronize()
        out[how] = {k: fs.download(k, n) for k in ("px", "py", "pz", "pflag")}
        fs.close()
    v = first["pflag"] == 2
    assert np.any(out["state"]["px"][v] != first["px"][v])   # the parcels were advected
    for k in ("px", "py", "pz"):
        assert np.allclose(out["state"][k][v], out["fields"][k][v], rtol=0, atol=1e-4), k
