"""G2P and advection: the variant for few particles (everything inline) and the
one for many (rare branches out of line, float velocities and near-rock map in
front of the double-precision tests) give every particle the same bits: the
pass over all particles against passes over a leading part of them, on both
sides of the line (148 * 256), for water, spray, ice, cooled particles and
particles inside rock and beyond the shell."""
import numpy as np
import pytest

from fluid_solver import FluidSolver

pytestmark = pytest.mark.gpu
LINE = 148 * 256
KEYS = ("px", "py", "pz", "pvx", "pvy", "pvz", "pflag", "pcool", "pAir")


@pytest.mark.parametrize("n,dx", [(48, 1.0), (45, 0.9)])
def test_variants_agree(n, dx):
    R, depth = 0.4 * n * dx, 0.1 * n * dx
    fs = FluidSolver(nx=n, ny=n, nz=n, dx=dx, coreR=R - depth, terrainSeed=5, targetParticles=120000.0, capacity=300000)
    fs.generateTerrain(5, R)
    fs.resetWater(depth)
    nP = fs.scalars.nP
    assert nP > LINE + 100
    fs.set_params(pic=0.05, maxSpeed=3.0, thermalOn=0, sorTol=0.0, pressureIters=5)
    fs.set_scalars(gRamp=1.5)
    fs._substep(0.01)
    fs.synchronize()
    r = np.random.default_rng(n)
    c = np.float32(0.5 * n * dx)
    pos = {k: fs.download(k)[:nP] for k in ("px", "py", "pz")}
    move = r.random(nP) < 0.1                          # spread over the rock, the sky and beyond the shell
    s = (r.uniform(0.3, 1.3, nP) ** 1.0).astype(np.float32)
    for k in pos:
        pos[k] = np.where(move, np.clip(c + (pos[k] - c) * s, 0.0, n * dx), pos[k]).astype(np.float32)
        fs.upload(k, pos[k])
    for k in ("pvx", "pvy", "pvz"):
        fs.upload(k, r.normal(scale=1.2, size=nP).astype(np.float32))
    fs.upload("pflag", r.choice(np.array([0, 1, 4, 5], np.uint8), nP, p=[0.88, 0.06, 0.03, 0.03]))
    fs.upload("pcool", (r.random(nP) < 0.05).astype(np.uint8))
    for k in ("u", "v", "w", "uO", "vO", "wO"):
        fs.upload(k, r.normal(scale=0.4, size=fs.field_size(k)).astype(np.float32))
    snap = {k: fs.download(k)[:nP] for k in KEYS}

    def run(count):
        for k, a in snap.items():
            fs.upload(k, a)
        fs.set_nparticles(count)
        fs.stage("G2P_ADVECT", 0.01)
        out = {k: fs.download(k)[:count] for k in KEYS}
        fs.set_nparticles(nP)
        return out

    every = run(nP)
    for k in KEYS:
        assert k == "pAir" or np.any(every[k] != snap[k]), k
    for count in (1, 33, LINE, LINE + 1, LINE + 100):
        part = run(count)
        for k in KEYS:
            assert np.array_equal(part[k].view(np.uint8), every[k][:count].view(np.uint8)), (k, count)
    fs.close()
