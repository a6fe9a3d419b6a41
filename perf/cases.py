"""The work that a program on this library has it do, as cases that can be timed and checked.

Every case is a planet: voxel terrain on the (2 n)^3 lattice around a sphere,
an ocean up to the sea-level radius, particles on a jittered lattice in the
water (x fastest, as the library's own fill lays them), and tangential
currents. A pass starts from host data wherever the library keeps state
between calls, so every pass on one state computes the same thing: it uploads
the particles and the last pressure, advances the planet, and reads the
particles back, as a host that drives the solver and draws from its own
arrays does.

kinds
  substep   `substeps` FLIP/MAC substeps: upload_state, _substep, download_state
  learned   the same with the learned warm start of the pressure solve on
  frame     whole 60 Hz frames with the thermal cycle on (FluidSolver.step)
  train     the gradients of `samples` training pairs (unet_accumulate), the
            half of a training step before the update or the all-reduce
  skin      the metaball surface of the particles, into vertex buffers on the GPU
  hud       the reductions a display shows every frame (energy, census)
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.getcwd(), "watersim-v1_b200"))
from fluid_solver import FluidSolver  # noqa: E402

DT = 0.01                     # the reference's substep of step(1/60)
MOVING = ("px", "py", "pz", "pvx", "pvy", "pvz", "pflag")
THERMAL = MOVING + ("pcool", "pT", "pAir", "pLight", "pDepth", "pWx", "pWy", "pWz", "pPh")
PLAIN = dict(pic=0.05, omega=1.7, maxSpeed=3.2, cfl=3.0, viscosity=5e-4, thermalOn=0)


def listed():
    return [
        # the smallest planet of the tests and examples, ~10k particles, the reference's fixed 40
        # iterations: every call is launches and waits
        dict(name="substep_32", kind="substep", n=32, R=12.0, depth=3.0, particles=10000, substeps=1, iters=40),
        # an odd grid: partial bricks along each axis, no aligned rows
        dict(name="substep_97", kind="substep", n=97, R=39.5, depth=6.5, particles=700000, substeps=4, iters=40),
        # the benchmark planet, solved to a residual of 1e-5
        dict(name="substep_128", kind="substep", n=128, R=52.0, depth=8.0, particles=1860000, substeps=10, iters=0),
        # the large planet of the benchmark, above the shared-memory solve's grids
        dict(name="substep_256", kind="substep", n=256, R=110.0, depth=12.0, particles=15300000, substeps=6, iters=0),
        # the benchmark planet with every solve started from the network's prediction
        dict(name="learned_128", kind="learned", n=128, R=52.0, depth=8.0, particles=1860000, substeps=10),
        # an application's frames: heat, evaporation, vapour and ice contacts around the substeps;
        # three frames hold one thermal tick (25 Hz at 60 frames per second)
        dict(name="frame_64", kind="frame", n=64, R=26.0, depth=5.0, particles=193000, vapour=4000, frames=3),
        # one batch of the warm start's training at the benchmark's size
        dict(name="train_128", kind="train", n=128, R=52.0, depth=8.0, samples=4),
        # the skin of a small and of the benchmark planet at the app's default tension
        dict(name="skin_48", kind="skin", n=48, R=19.5, depth=4.0, particles=60000, tension=0.5, detail=1.0),
        dict(name="skin_128", kind="skin", n=128, R=52.0, depth=8.0, particles=1860000, tension=0.5, detail=1.0),
        # what the display polls beside the picture
        dict(name="hud_128", kind="hud", n=128, R=52.0, depth=8.0, particles=1860000),
    ]


def draw(rng):
    kind = rng.choice(["substep", "substep", "substep", "learned", "frame", "train", "skin", "hud"])
    lo, hi = {"substep": (24, 200), "learned": (32, 144), "frame": (32, 112), "train": (24, 136), "skin": (24, 136),
              "hud": (24, 200)}[kind]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    R = round(n * rng.uniform(0.39, 0.425), 2)
    depth = round(max(2.5, R * rng.uniform(0.12, 0.3)), 2)
    # mean water column about 0.32 of the depth (_terrain), 8 to 24 particles per water cell
    water = 4 * math.pi * R * R * 0.32 * depth
    particles = int(min(15e6, water * rng.uniform(8, 24)))
    c = dict(kind=kind, n=n, R=R, depth=depth)
    if kind == "train":
        return dict(c, samples=rng.randint(1, 4))
    c["particles"] = particles
    if kind == "substep":
        return dict(c, substeps=rng.randint(1, 6), iters=rng.choice([0, 20, 40, rng.randint(10, 60)]))
    if kind == "learned":
        return dict(c, substeps=rng.randint(2, 8))
    if kind == "frame":
        return dict(c, vapour=int(particles * rng.uniform(0.0, 0.04)), frames=3)
    if kind == "skin":
        return dict(c, tension=round(rng.uniform(0.2, 0.8), 2), detail=round(rng.uniform(0.6, 1.3), 2))
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _waves(seed, salt, count, low, high):
    """Random plane waves: wave vectors of `low`..`high` radians per unit length, phases, amplitudes ~ 1/|k|."""
    r = np.random.default_rng([int(seed), salt])
    d = r.normal(size=(count, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    k = np.exp(r.uniform(math.log(low), math.log(high), count))
    a = 1 / k
    a *= math.sqrt(2 / np.sum(a * a))          # unit variance of the sum
    return d * k[:, None], r.uniform(0, 2 * math.pi, count), a


def _terrain(case, seed):
    """The voxel terrain: the rock radius along each voxel's direction (land on about 29% of the
    sphere, basins to 1.4 depths below the sea) and the rock mask."""
    n, Rs, depth = case["n"], case["R"], case["depth"]
    m, dv = 2 * n, 0.5
    k, ph, a = _waves(seed, 1, 18, 1.5, 10.0)
    p = (torch.arange(m, device="cuda", dtype=torch.float32) + 0.5) * dv - n / 2
    X, Y = p[None, :], p[:, None]
    R = torch.empty(m, m, m, device="cuda")
    solid = torch.empty(m, m, m, dtype=torch.uint8, device="cuda")
    for z in range(m):
        r = torch.sqrt(X * X + Y * Y + p[z] * p[z])
        h = torch.zeros_like(r)
        for q in range(len(a)):
            h += float(a[q]) * torch.cos((float(k[q, 0]) * X + float(k[q, 1]) * Y + float(k[q, 2]) * p[z]) / r + float(ph[q]))
        R[z] = Rs + depth * torch.clamp(-0.25 + 0.45 * h, -1.4, 1.0)
        solid[z] = (r <= R[z]).to(torch.uint8)
    return dict(n=m, dv=dv, Rsl=Rs, Rlo=float(R.min()), Rhi=float(R.max()), landFrac=0.29, solid=solid, R=R)


def _rock(t, x, y, z, n):
    """Rock at the cell of each point (the voxel at the cell's centre), cells clamped off the shell."""
    i, j, k = (torch.clamp(v.to(torch.int64), 1, n - 2) * 2 + 1 for v in (x, y, z))
    return t["solid"].view(-1)[(k * t["n"] + j) * t["n"] + i] == 1


def _lattice(case, t, s, g):
    """The jittered lattice of spacing s in the water, x fastest, then z, then y."""
    n, Rs = case["n"], case["R"]
    axis = torch.arange(-Rs, Rs, s, device="cuda", dtype=torch.float32)
    rows = max(1, 2000000 // len(axis) ** 2)
    lo2, hi2 = (t["Rlo"] - s) ** 2, (Rs - 0.4 * s) ** 2
    parts = []
    for a in range(0, len(axis), rows):
        y, z, x = torch.meshgrid(axis[a:a + rows], axis, axis, indexing="ij")
        r2 = x * x + y * y + z * z
        at = ((r2 > lo2) & (r2 < hi2)).reshape(-1).nonzero().squeeze(1)
        q = torch.stack([x.reshape(-1)[at], y.reshape(-1)[at], z.reshape(-1)[at]])
        q += n / 2 + (torch.rand(q.shape, generator=g, device="cuda") - 0.5) * 0.3 * s
        v = torch.clamp((q * 2).to(torch.int64), 0, t["n"] - 1)
        rock = _rock(t, *q, n) | (t["solid"].view(-1)[(v[2] * t["n"] + v[1]) * t["n"] + v[0]] == 1)
        parts.append(q[:, ~rock])
    return torch.cat(parts, 1)


def _planet(case, seed):
    """Terrain, particles (float32, on the GPU) and their spacing."""
    n, Rs = case["n"], case["R"]
    t = _terrain(case, seed)
    c = n / 2
    p = (torch.arange(t["n"], device="cuda", dtype=torch.float32) + 0.5) * 0.5 - c
    water = 0
    for z in range(0, t["n"], 4):
        r2 = (p * p)[None, :] + (p * p)[:, None] + p[z] * p[z]
        water = water + ((t["solid"][z] == 0) & (r2 < Rs * Rs)).sum()
    s, P = (int(water) * 4 * 0.125 / (1.06 * case["particles"])) ** (1 / 3), case["particles"]
    g = _gen(seed, 2)
    for _ in range(4):
        pos = _lattice(case, t, s, g)
        if pos.shape[1] >= P:
            break
        s *= 0.995 * (max(1, pos.shape[1]) / P) ** (1 / 3)
    # exactly the asked number: the few sites too many are left out evenly
    N = pos.shape[1]
    if N < P:
        raise ValueError("the water holds %d lattice sites of spacing %g, fewer than %d" % (N, s, P))
    pos = pos[:, torch.arange(P, device="cuda") * N // P].contiguous()
    # currents: tangential, smooth over a quarter of the planet down to a few cells, about 0.4 m/s
    k, ph, a = _waves(seed, 3, 10, 4 / Rs, 40 / Rs)
    e = pos - c
    rad = torch.linalg.norm(e, dim=0)
    w = torch.zeros_like(e)
    for q in range(len(a)):
        arg = float(k[q, 0]) * e[0] + float(k[q, 1]) * e[1] + float(k[q, 2]) * e[2] + float(ph[q])
        w[q % 3] += 0.4 * float(a[q]) * torch.cos(arg)
    vel = torch.cross(w, e / rad, dim=0) + 0.02 * torch.randn(e.shape, generator=g, device="cuda")
    return t, pos, vel, s


def _hydrostatic(case, dt):
    """The pressure of a resting ocean in the solver's units: gravity * dt per cell of depth below the sea."""
    n, Rs = case["n"], case["R"]
    p = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) - n / 2
    r = torch.sqrt(p[:, None, None] ** 2 + p[None, :, None] ** 2 + p[None, None, :] ** 2)
    return (9.81 * dt * Rs * torch.clamp(Rs / torch.clamp(r, min=1.0) - 1, min=0)).to(torch.float32).reshape(-1)


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype).pin_memory()
    h.copy_(t)
    return h.numpy()


def _solver(case, t, spacing, nP, capacity=None, **params):
    n = case["n"]
    fs = FluidSolver(nx=n, ny=n, nz=n, dx=1.0, coreR=case["R"] - case["depth"], targetParticles=float(max(1, nP)),
                     capacity=capacity or nP + 8192, device=0)
    fs.upload_terrain(dict(t, solid=t["solid"].reshape(-1).cpu().numpy(), R=t["R"].reshape(-1).cpu().numpy()))
    fs.set_params(**params)
    fs.set_scalars(oceanR=case["R"], spacing=spacing, particleVolume=spacing ** 3, gRamp=1.5, nP=nP)
    return fs


def _solve_params(iters):
    return dict(sorTol=0.0, pressureIters=iters) if iters else dict(sorTol=1e-5, sorCheckEvery=10, sorMaxIters=5000)


def _net_weights(seed):
    """He-normal weights of the 3-level network, flat as unet_set_weights takes them."""
    r = np.random.default_rng([int(seed), 4])
    out = []
    for cin, cout in NET:
        out += [r.normal(0, math.sqrt(2 / (27 * cin)), cout * cin * 27), r.normal(0, 0.02, cout)]
    return np.concatenate(out + [r.normal(0, 0.25, 16), np.zeros(1)]).astype(np.float32)


# (input, output channels) of e0a e0b e1a e1b ba bb d1a d1b d0a d0b
NET = ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16))


def _cell_types(case, t):
    """0 air, 1 water, 2 rock of a resting ocean, (n, n, n) with the domain's shell closed."""
    n = case["n"]
    solid = t["solid"][1::2, 1::2, 1::2] == 1
    p = (torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) - n / 2
    r2 = p[:, None, None] ** 2 + p[None, :, None] ** 2 + p[None, None, :] ** 2
    ty = torch.where(solid, 2, torch.where(r2 < case["R"] ** 2, 1, 0)).to(torch.uint8)
    for a in range(3):
        ty.select(a, 0).fill_(2)
        ty.select(a, n - 1).fill_(2)
    return ty


def _pairs(case, seed):
    """Training pairs: the resting ocean's cell types, a rough residual of unit RMS and a smooth correction."""
    n = case["n"]
    ty = _cell_types(case, _terrain(case, seed))
    g = _gen(seed, 5)
    p = torch.arange(n, device="cuda", dtype=torch.float32)
    for s in range(case["samples"]):
        k, ph, a = _waves(seed, 100 + s, 6, 0.05, 0.8)
        target = torch.zeros(n, n, n, device="cuda")
        for q in range(6):
            target += float(a[q]) * torch.cos(float(k[q, 0]) * p + float(k[q, 1]) * p[:, None] +
                                              float(k[q, 2]) * p[:, None, None] + float(ph[q]))
        fluid = (ty == 1).float()
        yield torch.randn(n, n, n, generator=g, device="cuda") * fluid, ty, target * fluid


def _atmosphere(case, seed, t, pos, vel):
    """The particle fields of a planet whose thermal cycle has run for a while: sun-warmed water,
    `vapour` parcels (steam, cloud, a little rain) under the sky, ice at the cold poles."""
    g = _gen(seed, 6)
    c, m, Rs = case["n"] / 2, case["vapour"], case["R"]
    rand = lambda *s: torch.rand(s, generator=g, device="cuda")  # noqa: E731
    d = torch.randn(3, m, generator=g, device="cuda")
    d /= torch.linalg.norm(d, dim=0)
    pos = torch.cat([pos, c + d * (Rs + 0.16 + 0.17 * rand(m))], 1)
    vel = torch.cat([vel, torch.cross(d, torch.randn(3, m, generator=g, device="cuda"), dim=0)], 1)
    nP = pos.shape[1]
    nW = nP - m
    e = (pos - c) / torch.linalg.norm(pos - c, dim=0)
    lit = torch.clamp(e[0], min=0)
    f = {k: torch.zeros(nP, device="cuda") for k in THERMAL if k not in ("pflag", "pcool", "pDepth")}
    f["px"], f["py"], f["pz"] = pos
    f["pvx"], f["pvy"], f["pvz"] = vel
    f["pT"] = 0.16 + 0.42 * lit + 0.04 * rand(nP)
    flag = torch.zeros(nP, dtype=torch.uint8, device="cuda")
    pick = rand(nP)
    flag[nW:] = torch.where(pick[nW:] < 0.7, 2, torch.where(pick[nW:] < 0.95, 3, 4)).to(torch.uint8)
    f["pT"][nW:] = 0.23 + 0.2 * pick[nW:]
    ice = (e[1, :nW].abs() > 0.97) & (torch.linalg.norm(pos[:, :nW] - c, dim=0) > Rs - 0.8)
    flag[:nW][ice] = 5
    f["pAir"][:nW][ice] = 1.0
    f["pT"][:nW][ice] = 0.06
    f["pAir"][nW:] = 2 * rand(m)
    f["pLight"] = lit.clone()
    f["pflag"] = flag
    f["pcool"] = torch.zeros(nP, dtype=torch.uint8, device="cuda")
    f["pDepth"] = torch.zeros(nP, dtype=torch.uint8, device="cuda")
    return f


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        t = dict(n=2, dv=case["n"] / 2, Rsl=case["R"], Rlo=1.0, Rhi=1.0, landFrac=0.0,
                 solid=torch.zeros(8, dtype=torch.uint8), R=torch.ones(8))
        fs = _solver(case, t, 0.5, 0, **PLAIN)
        fs.unet_init(1, 3)
        fs.unet_set_weights(_net_weights(seed))
        fs.unet_set_gain(1.0)
        fs.unet_collect(case["samples"])
        fs.unet_collect(0)
        for r0, ty, target in _pairs(case, seed):
            fs.unet_put_pair(r0.reshape(-1).cpu().numpy(), ty.reshape(-1).cpu().numpy(), target.reshape(-1).cpu().numpy())
        grads = fs.unet_grads()
        grads.owner = fs                             # the solver owns the memory the tensor shows
        return dict(kind=kind, fs=fs, samples=case["samples"], grads=grads)
    t, pos, vel, s = _planet(case, seed)
    nP = pos.shape[1]
    if kind in ("substep", "learned"):
        fs = _solver(case, t, s, nP, **PLAIN, **_solve_params(case.get("iters", 0)))
        if kind == "learned":
            fs.unet_init(1, 3)
            fs.unet_set_weights(_net_weights(seed))
            fs.unet_set_gain(0.02)
            fs.unet_enable(True)
        dev = dict(zip(MOVING[:6], [*pos, *vel]), pflag=torch.zeros(nP, dtype=torch.uint8))
        host = {k: _pinned(v) for k, v in dev.items()}
        return dict(kind="substep", fs=fs, nP=nP, host=host, q=_pinned(_hydrostatic(case, DT)),
                    out={k: _pinned(torch.zeros_like(v)) for k, v in dev.items()}, substeps=case["substeps"])
    if kind == "frame":
        f = _atmosphere(case, seed, t, pos, vel)
        nP += case["vapour"]
        c = case["n"] / 2
        fs = _solver(case, t, s, nP, **dict(PLAIN, thermalOn=1), vorticity=0.05, sunActivity=0.6, evapIntensity=0.05,
                     sunPos=[c + 3 * case["R"] * math.cos(0.408), c + 3 * case["R"] * math.sin(0.408), c],
                     **_solve_params(0))
        # what the passes before the first substep read: the last frame's cell types, face velocities and density
        n = case["n"]
        faces = n * n * (n + 1)
        dens = torch.nn.functional.pad((_cell_types(case, t) == 1).float(), (0, 1, 0, 1, 0, 1)) * 2.5
        grid = dict(cellType=_pinned(_cell_types(case, t).reshape(-1)), u=_pinned(torch.zeros(faces)),
                    v=_pinned(torch.zeros(faces)), w=_pinned(torch.zeros(faces)), dens=_pinned(dens.reshape(-1)),
                    q=_pinned(_hydrostatic(case, DT)))
        return dict(kind=kind, fs=fs, nP=nP, host={k: _pinned(v) for k, v in f.items()}, grid=grid,
                    out={k: _pinned(torch.zeros_like(v)) for k, v in f.items()}, frames=case["frames"],
                    scalars=dict(simTime=10.0, heatAcc=1 / 25.0, evS=0x51ab3c77, cfS=0x2f6e2b1, bfS=0x7f4a7c15))
    fs = _solver(case, t, s, nP, **PLAIN)
    for k, v in zip(MOVING, [*pos, *vel, torch.zeros(nP, dtype=torch.uint8)]):
        if kind == "hud" and k == "pflag":           # a display of a planet with some vapour and ice
            v = _hud_flags(nP, seed)
        fs.upload(k, v.cpu().numpy())
    if kind == "hud":
        return dict(kind=kind, fs=fs)
    return dict(kind=kind, fs=fs, tension=case["tension"], detail=case["detail"],
                pos=torch.zeros(_skin_room(case), 3, device="cuda"), nrm=torch.zeros(_skin_room(case), 3, device="cuda"))


def _skin_room(case):
    """Vertices that a drawing program makes room for: about 40 come for each square cell of the sphere."""
    return int(100 * 4 * math.pi * (case["R"] * case["detail"]) ** 2)


def _hud_flags(nP, seed):
    r = torch.rand(nP, generator=_gen(seed, 7), device="cuda")
    return torch.where(r < 0.9, 0, torch.where(r < 0.93, 1, torch.where(r < 0.96, 2, torch.where(r < 0.98, 3, 5)))).to(torch.uint8)


# ---------------------------------------------------------------- run
class _View:
    """A float32 device buffer of a solver, which lives as long as the view."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3, "strides": None}


def run(state):
    fs = state["fs"]
    kind = state["kind"]
    if kind == "substep":
        fs.upload("q", state["q"])
        fs.upload_state(state["host"], state["nP"])
        for _ in range(state["substeps"]):
            fs._substep(DT)
        fs.download_state(state["out"], state["nP"])
        return state["out"]
    if kind == "frame":
        fs.set_scalars(**state["scalars"])
        for k, v in state["grid"].items():
            fs.upload(k, v)
        fs.upload_state(state["host"], state["nP"])
        for _ in range(state["frames"]):
            fs.step(1 / 60)
        fs.download_state(state["out"], state["nP"])
        return state["out"]
    if kind == "train":
        loss = fs.unet_accumulate(state["samples"], 11)
        return {"loss": loss, "grads": state["grads"]}
    if kind == "skin":
        count, vol = C.c_int64(), C.c_double()
        L, h = fs._L, fs._h
        fs._check(L.ws_metaball_mesh(h, state["tension"], state["detail"], C.byref(count), C.byref(vol)))
        pos, nrm = C.c_void_p(), C.c_void_p()
        fs._check(L.ws_metaball_device(h, C.byref(pos), C.byref(nrm), C.byref(count)))
        for k, p in (("pos", pos), ("nrm", nrm)):   # into the drawing program's vertex buffers
            state[k][:count.value].copy_(torch.as_tensor(_View(fs, p.value, (count.value, 3)), device="cuda:0"))
            state[k][count.value:].zero_()
        return {"volume": vol.value, "vertices": count.value, "pos": state["pos"], "nrm": state["nrm"]}
    return {"energy": fs.kineticEnergy(), "census": fs.census()}


# ---------------------------------------------------------------- work
def work(case):
    """What one pass cannot do without. Per substep: the moving fields of each particle in and out
    (50 bytes), pressure, right-hand side and stencil of each water cell; about 400 operations per
    particle for the two transfers and 15 per water cell and iteration (60 where the solve stops
    at a residual). The fields a pass uploads and reads back are counted with the substeps'."""
    kind, R, depth = case["kind"], case["R"], case["depth"]
    water = 4 * math.pi * R * R * 0.32 * depth
    P = case.get("particles", 0) + case.get("vapour", 0)
    # multiply-adds of the network per voxel of each level (27 taps), active tiles about 2.5x the water
    net = 2.5 * water * 27 * (256 + 256 + 768 + 256 + (512 + 1024 + 3072 + 1024) / 8 + (2048 + 4096) / 64)
    if kind in ("substep", "learned"):
        K = case["substeps"]
        b, f = K * (50 * P + 13 * water), K * (400 * P + 15 * water * (case.get("iters") or 60))
        if kind == "learned":
            b, f = b + K * 2.5 * water * 2 * 16 * 2, f + K * 2 * net
        return {"bytes": b, "flops": f}
    if kind == "frame":
        K = 2 * case["frames"]
        return {"bytes": K * (50 * P + 13 * water) + 60 * P, "flops": K * (400 * P + 15 * water * 60) + 600 * P}
    if kind == "train":
        s = case["samples"]
        return {"bytes": s * 2.5 * water * (9 + 2 * 2 * 16 * 10), "flops": s * 3 * 2 * net}
    if kind == "skin":
        r = 1.6 + 2.2 * case["tension"]
        corners = (case["n"] * case["detail"]) ** 3
        touched = 4.19 * (r * (water / P) ** (1 / 3) * case["detail"]) ** 3
        return {"bytes": 13 * P + 4 * corners, "flops": 8 * P * touched}
    return {"bytes": 13 * P, "flops": 6 * P}


# ---------------------------------------------------------------- exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "substep" and case["iters"]:
        return _exact_substeps(case, seed)
    # Solves that stop at a residual have no value of their own: how far they stop is part of the
    # result. Frames walk three serial random streams particle by particle, which plain code
    # cannot do in 20 seconds.
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "skin":
        return _exact_skin(case, seed)
    if kind == "hud":
        t, pos, vel, s = _planet(case, seed)
        flag = _hud_flags(pos.shape[1], seed)
        count = [int(torch.isin(flag, torch.tensor(w, dtype=torch.uint8, device="cuda")).sum()) for w in ((0, 1, 4), (5,), (2, 3))]
        return {"energy": float(500 * s ** 3 * vel.double().square().sum()),
                "census": tuple(c / sum(count) for c in count)}
    return None


def _along(v, axis, lo, hi):
    return v.narrow(axis, lo, hi - lo)


def _exact_substeps(case, seed):
    """The FLIP/MAC substep in 64 bits: arrays are (z, y, x), component c's faces have one more along
    its axis (axis 2 - c). The passes are short enough that no particle leaves the water."""
    n, Rs, K = case["n"], case["R"], case["substeps"]
    t, pos, vel, s = _planet(case, seed)
    x, v = pos.double(), vel.double()
    c, dom = n / 2, n / 2 - 1
    dev = x.device
    D = dict(dtype=torch.float64, device=dev)
    static = torch.where(_cell_types(case, t) == 2, 2, 0)
    q = _hydrostatic(case, DT).double()
    p = torch.arange(n, **D) + 0.5 - c
    edge = torch.arange(n + 1, **D) - c
    shape = [[n + (a == 2 - d) for a in range(3)] for d in range(3)]
    lim = torch.tensor([n - 1, n - 2, n - 2], device=dev)
    half = lambda d: torch.tensor([0.0 if a == d else 0.5 for a in range(3)], **D)[:, None]  # noqa: E731

    def stencil(d, X):
        a = X - half(d)
        i = torch.floor(a)
        f = torch.where(i < 0, 0.0, torch.where(i > lim[:, None], 1.0, a - i))
        i = torch.minimum(torch.clamp(i, min=0), lim[:, None].double()).to(torch.int64)
        _, ny, nx = shape[d]
        base = (i[2] * ny + i[1]) * nx + i[0]
        for b in range(8):
            o = (b & 1, b >> 1 & 1, b >> 2)
            w = 1
            for ax in range(3):
                w = w * (f[ax] if o[ax] else 1 - f[ax])
            yield base + (o[2] * ny + o[1]) * nx + o[0], w

    def sample(u, X):
        return torch.stack([sum(u[d].view(-1)[at] * w for at, w in stencil(d, X)) for d in range(3)])

    def sides(d, a):          # the cells left and right of component d's inner faces
        ax = 2 - d
        return _along(a, ax, 0, n - 1), _along(a, ax, 1, n)

    def inner(d, a):
        return _along(a, 2 - d, 1, n)

    for _ in range(K):
        cell = torch.clamp(torch.floor(x), 0, n - 1).to(torch.int64)
        cell = (cell[2] * n + cell[1]) * n + cell[0]
        ty = static.clone().view(-1)
        ty[cell] = torch.where(ty[cell] == 0, 1, ty[cell])
        ty = ty.view(n, n, n)
        u, uo, valid, opened = [], [], [], []
        for d in range(3):
            m = torch.zeros(shape[d], **D)
            w = torch.zeros(shape[d], **D)
            for at, wt in stencil(d, x):
                m.view(-1).index_add_(0, at, wt * v[d])
                w.view(-1).index_add_(0, at, wt)
            m = torch.where(w > 1e-8, m / torch.where(w > 0, w, 1.0), m)
            l, r = sides(d, ty)
            free = torch.zeros(shape[d], dtype=torch.bool, device=dev)
            inner(d, free).copy_((l != 2) & (r != 2))
            m = torch.where(free, m, 0.0)
            valid.append((w > 1e-8) | ~free)
            opened.append(free)
            uo.append(m)
            wet = torch.zeros_like(free)
            inner(d, wet).copy_((l == 1) | (r == 1))
            both = torch.zeros_like(free)
            inner(d, both).copy_((l == 1) & (r == 1))
            lap = 6 * m
            for a in range(3):
                k = shape[d][a]
                lap = lap - torch.cat([_along(m, a, 0, 1), _along(m, a, 0, k - 1)], a)
                lap = lap - torch.cat([_along(m, a, 1, k), _along(m, a, k - 1, k)], a)
            e = [(edge if a == 2 - d else p).view([-1 if a == b else 1 for b in range(3)]) for a in range(3)]
            r3 = (e[0] ** 2 + e[1] ** 2 + e[2] ** 2) ** 1.5
            grav = -Rs * Rs * e[2 - d] / torch.where(r3 == 0, 1e-9, r3)
            un = m + torch.where(both, 5e-4 * DT * lap, 0.0) + torch.where(wet, grav * DT * 9.81, 0.0)
            u.append(torch.where(free, un, 0.0))
        fluid = ty == 1
        div = sum(_along(u[d], 2 - d, 1, n + 1) - _along(u[d], 2 - d, 0, n) for d in range(3))
        diag = torch.zeros(n, n, n, **D)
        for a in range(3):
            _along(diag, a, 0, n - 1).add_(_along(ty, a, 1, n) != 2)
            _along(diag, a, 1, n).add_(_along(ty, a, 0, n - 1) != 2)
        q = torch.where(fluid.view(-1), q, 0.0)
        i = torch.arange(n, device=dev)
        colour = (i[:, None, None] + i[None, :, None] + i[None, None, :]) & 1
        lists = [(fluid & (colour == k)).view(-1).nonzero().squeeze(1) for k in (0, 1)]
        parts = [(at, 1.7 / diag.view(-1)[at], -div.reshape(-1)[at]) for at in lists]
        for _ in range(case["iters"]):
            for at, pw, b in parts:
                nb = q[at - 1] + q[at + 1] + q[at - n] + q[at + n] + q[at - n * n] + q[at + n * n]
                q[at] = q[at] * (1 - 1.7) + pw * (b + nb)
        q3 = q.view(n, n, n)
        for d in range(3):
            l, r = sides(d, q3)
            g = torch.zeros(shape[d], **D)
            inner(d, g).copy_(r - l)
            u[d] = torch.clamp(torch.where(opened[d], u[d] - g, u[d]), -3.2 * 1.1, 3.2 * 1.1)
            tot, cnt = torch.zeros(shape[d], **D), torch.zeros(shape[d], **D)
            ok = valid[d].double()
            for a in range(3):
                k = shape[d][a]
                for dst, src in (((0, k - 1), (1, k)), ((1, k), (0, k - 1))):
                    _along(tot, a, *dst).add_(_along(u[d] * ok, a, *src))
                    _along(cnt, a, *dst).add_(_along(ok, a, *src))
            u[d] = torch.where(~valid[d] & (cnt > 0), tot / torch.clamp(cnt, min=1), u[d])
        now, old = sample(u, x), sample(uo, x)
        v = (v + now - old) * (1 - 0.05) + now * 0.05
        v = v * torch.clamp(3.2 / torch.linalg.norm(v, dim=0).clamp(min=1e-30), max=1.0)
        mid = torch.clamp(x + 0.5 * DT * now, 1.02, n - 1.02)
        adv = torch.where((now * now).sum(0) > 0.25, sample(u, mid), now)
        cut = torch.clamp(3.2 / torch.linalg.norm(adv, dim=0).clamp(min=1e-30), max=1.0)
        adv, v = adv * cut, v * cut
        x = x + adv * DT
        out = x - c
        r = torch.linalg.norm(out, dim=0)
        up = out / r
        tried = torch.zeros(x.shape[1], dtype=torch.bool, device=dev)
        for _ in range(8):
            hit = _rock(t, *x, n).nonzero().squeeze(1)
            tried[hit] = True
            step = torch.clamp(dom - 0.02 - torch.linalg.norm(x[:, hit] - c, dim=0), max=0.5)
            x[:, hit] += up[:, hit] * step
        hit = tried.nonzero().squeeze(1)
        if len(hit):
            xs = x[:, hit]
            e = xs - c
            er = torch.linalg.norm(e, dim=0)
            want = _terrain_radius(t, xs) + 0.06
            xs = torch.where(er > want, c + e / er * want, xs)
            for _ in range(4):
                xs = xs + torch.where(_rock(t, *xs, n), e / er * 0.5, 0.0)
            x[:, hit] = xs
            vr = (v[:, hit] * up[:, hit]).sum(0)
            v[:, hit] -= up[:, hit] * torch.clamp(vr, max=0)
        floor = tried | _rock(t, *(x - up), n)
        v = torch.where(floor, v * (1 - 0.6 * DT), v)
        e = x - c
        e = e / torch.linalg.norm(e, dim=0)
        v = (v - e * ((v * e).sum(0) * DT)) * (1 - 0.42 * DT)
    got = dict(zip(MOVING[:6], [*x, *v]), pflag=torch.zeros(x.shape[1], dtype=torch.uint8))
    return {k: a.cpu() for k, a in got.items()}


def _terrain_radius(t, X):
    """The trilinear terrain radius at points X (3, P)."""
    m = t["n"]
    g = X * 2 - 0.5
    i = torch.clamp(g.to(torch.int64), 0, m - 2)
    f = torch.clamp(g - i, 0, 1)
    R, out = t["R"].view(-1), 0
    for b in range(8):
        o = (b & 1, b >> 1 & 1, b >> 2)
        w = 1
        for a in range(3):
            w = w * (f[a] if o[a] else 1 - f[a])
        out = out + w * R[((i[2] + o[2]) * m + i[1] + o[1]) * m + i[0] + o[0]].double()
    return out


def _exact_train(case, seed):
    """The network, its loss and its gradients in 64 bits: activations are zero off the active tiles
    (8 x 16 x 8 voxels; at the finest level those with water, above those with an active child)."""
    n = case["n"]
    flat = torch.from_numpy(_net_weights(seed)).double().cuda()
    pairs = list(_pairs(case, seed))
    sizes = [n, (n + 1) // 2, ((n + 1) // 2 + 1) // 2]
    tiles = [[-(-s // 8), -(-s // 16), -(-s // 8)] for s in sizes]
    act = F.max_pool3d(F.pad((pairs[0][1] == 1).float()[None, None],
                             (0, tiles[0][2] * 8 - n, 0, tiles[0][1] * 16 - n, 0, tiles[0][0] * 8 - n)), (8, 16, 8))
    acts = [act]
    for lv in (1, 2):
        a = F.pad(acts[-1], [w for k in (2, 1, 0) for w in (0, 2 * tiles[lv][k] - tiles[lv - 1][k])])
        acts.append(F.max_pool3d(a, 2))
    mask = []
    for s, a in zip(sizes, acts):
        for k, w in ((2, 8), (3, 16), (4, 8)):
            a = a.repeat_interleave(w, k)
        mask.append(a[:, :, :s, :s, :s].double())
    params, at = [], 0
    for cin, cout in NET:
        for shape in ((cout, cin, 3, 3, 3), (cout,)):
            size = math.prod(shape)
            params.append(flat[at:at + size].view(shape).clone().requires_grad_())
            at += size
    params += [flat[at:at + 16].clone().requires_grad_(), flat[at + 16:at + 17].clone().requires_grad_()]

    def conv(l, a, lv):
        return F.relu(F.conv3d(a, params[2 * l], params[2 * l + 1], padding=1)) * mask[lv]

    def pool(a, lv):
        odd = sizes[lv] % 2
        return F.avg_pool3d(F.pad(a, (0, odd) * 3), 2) * mask[lv + 1]

    def up(a, lv):
        return F.interpolate(a, scale_factor=2, mode="nearest")[:, :, :sizes[lv], :sizes[lv], :sizes[lv]] * mask[lv]

    # the pairs the library draws for seed 11: a 64-bit linear congruential generator's upper 31 bits
    mul, inc, top = 6364136223846793005, 1442695040888963407, (1 << 64) - 1
    state, total = (11 * mul + inc) & top, 0.0
    for _ in range(case["samples"]):
        state = (state * mul + inc) & top
        r0, ty, target = pairs[(state >> 33) % len(pairs)]
        x = torch.stack([r0.double(), *((ty == k).double() for k in (1, 2, 0))])[None]
        x = F.pad(x, (0, 0, 0, 0, 0, 0, 0, 12)) * mask[0]
        s0 = conv(1, conv(0, x, 0), 0)
        s1 = conv(3, conv(2, pool(s0, 0), 1), 1)
        b = conv(5, conv(4, pool(s1, 1), 2), 2)
        d1 = conv(7, conv(6, torch.cat([up(b, 1), s1], 1), 1), 1)
        h = conv(9, conv(8, torch.cat([up(d1, 0), s0], 1), 0), 0)
        o = (h[0] * params[-2].view(16, 1, 1, 1)).sum(0) + params[-1]
        loss = ((o - target.double()) ** 2)[ty == 1].mean()
        loss.backward()
        total += float(loss)
        del x, s0, s1, b, d1, h, o, loss
    return {"loss": total, "grads": torch.cat([a.grad.reshape(-1) for a in params]).cpu()}


CORNERS = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
TETS = ((0, 5, 1, 6), (0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6))
EDGES = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))
# the triangles of each code (which of a tet's corners are inside), by edge
FACES = ((), ((0, 2, 3),), ((0, 1, 4),), ((2, 3, 4), (2, 4, 1)), ((2, 1, 5),), ((0, 3, 5), (0, 5, 1)), ((0, 4, 5), (0, 5, 2)),
         ((3, 5, 4),), ((3, 4, 5),), ((0, 2, 5), (0, 5, 4)), ((0, 1, 5), (0, 5, 3)), ((2, 1, 5),), ((2, 1, 4), (2, 4, 3)),
         ((0, 1, 4),), ((0, 2, 3),), ())


def _exact_skin(case, seed):
    """The metaball field and its marching-tetrahedra surface in 64 bits, cells in index order."""
    t, pos, vel, s = _planet(case, seed)
    n, x = case["n"], pos.double()
    m = max(6, int(math.floor(n * case["detail"] + 0.5)))
    dx = n / m
    reach = (1.6 + 2.2 * case["tension"]) * s / dx
    iso = 1.5 * ((1.6 + 2.2 * case["tension"]) / 1.6) ** 1.5
    g = x / dx
    at = torch.floor(g + 0.5).to(torch.int64)
    rad = min(3, math.ceil(reach))
    f = torch.zeros((m + 1) ** 3, dtype=torch.float64, device=x.device)
    for k in range(-rad, rad + 1):
        for j in range(-rad, rad + 1):
            for i in range(-rad, rad + 1):
                o = at + torch.tensor([i, j, k], device=x.device)[:, None]
                d2 = ((o - g) ** 2).sum(0)
                w = torch.where((d2 < reach * reach) & (o >= 0).all(0) & (o <= m).all(0), (1 - d2 / reach ** 2) ** 2, 0.0)
                o = torch.clamp(o, 0, m)
                f.index_add_(0, (o[2] * (m + 1) + o[1]) * (m + 1) + o[0], w)
    f = f.view(m + 1, m + 1, m + 1)
    low = -F.max_pool3d(-f[None, None], 2, 1)[0, 0]
    high = F.max_pool3d(f[None, None], 2, 1)[0, 0]
    cells = ((low <= iso) & (high >= iso)).nonzero()[:, [2, 1, 0]]
    i = torch.arange(m + 1, device=x.device)
    hi, lo = torch.clamp(i + 1, max=m), torch.clamp(i - 1, min=0)
    grad = torch.stack([f[:, :, hi] - f[:, :, lo], f[:, hi] - f[:, lo], f[hi] - f[lo]], -1) / (2 * dx)
    corner = [cells + torch.tensor(c, device=x.device) for c in CORNERS]
    val = torch.stack([f[c[:, 2], c[:, 1], c[:, 0]] for c in corner], 1)
    gr = torch.stack([grad[c[:, 2], c[:, 1], c[:, 0]] for c in corner], 1)
    found = []
    for nt, tet in enumerate(TETS):
        code = sum((val[:, tet[c]] > iso).long() << c for c in range(4))
        for k in range(1, 15):
            own = (code == k).nonzero().squeeze(1)
            for e, face in enumerate(FACES[k]):
                P, N = [], []
                for ed in face:
                    a, b = (tet[q] for q in EDGES[ed])
                    va, vb = val[own, a], val[own, b]
                    w = torch.clamp(torch.where(vb != va, (iso - va) / torch.where(vb != va, vb - va, 1.0), 0.5), 0, 1)[:, None]
                    P.append((corner[a][own] + (corner[b][own] - corner[a][own]) * w) * dx)
                    g1 = -(gr[own, a] + (gr[own, b] - gr[own, a]) * w)
                    ln = torch.linalg.norm(g1, dim=1, keepdim=True)
                    N.append(g1 / torch.where(ln == 0, 1.0, ln))
                back = (torch.cross(P[1] - P[0], P[2] - P[0], dim=1) * (N[0] + N[1] + N[2])).sum(1, keepdim=True) < 0
                P = torch.stack([P[0], torch.where(back, P[2], P[1]), torch.where(back, P[1], P[2])], 1)
                N = torch.stack([N[0], torch.where(back, N[2], N[1]), torch.where(back, N[1], N[2])], 1)
                found.append((own * 12 + nt * 2 + e, P, N))
    order = torch.argsort(torch.cat([a for a, _, _ in found]))
    P, N = (torch.cat([a[k] for a in found])[order] for k in (1, 2))
    vol = (P[:, 0] * torch.cross(P[:, 1], P[:, 2], dim=1)).sum() / 6
    P, N = (F.pad(a.reshape(-1, 3), (0, 0, 0, _skin_room(case) - 3 * len(a))).cpu() for a in (P, N))
    return {"volume": abs(float(vol)), "vertices": None, "pos": P, "nrm": N}
