"""_iceContacts (js/solver.js:3290-3324) at the edges of its group sweep:
lists of two grains, a chain of contacts, one clump in which every grain
touches more grains than a list entry holds, many separate pairs, and list
lengths around a block of threads. Stuck flags and velocities are those of
the reference's serial sweep, bit for bit."""
import numpy as np
import pytest

from helpers import planet, to_device

pytestmark = pytest.mark.gpu


def _grains(kind, m, rad, rng):
    if kind == "chain":                       # each grain touches the next along x
        return np.stack([np.arange(m) * 0.8 * rad, np.zeros(m), np.zeros(m)], 1)
    if kind == "clump":                       # all within one contact radius
        return rng.uniform(0, 0.5 * rad, (m, 3))
    if kind == "pairs":                       # far pairs, interleaved along x
        at = rng.uniform(0, 6, (m // 2, 3)) * [0.2, 1, 1]
        return np.concatenate([at, at + 0.3 * rad])
    return rng.uniform(0, 40 * rad, (m, 3))   # "far": hardly any contact


@pytest.mark.parametrize("kind,m", [("clump", 2), ("chain", 3), ("chain", 129), ("clump", 127), ("clump", 300),
                                    ("pairs", 256), ("far", 128), ("far", 1)])
def test_ice_groups_bitwise(kind, m):
    o = planet("planet32", thermalOn=1)
    nP = o.nP
    rng = np.random.default_rng(m)
    rad = o.scalars.spacing * 0.7
    sel = rng.choice(nP, m, replace=False)
    pos = 8.0 + _grains(kind, m, rad, rng)[rng.permutation(m)]
    for a, k in enumerate(("px", "py", "pz")):
        o.arr(k)[sel] = pos[:, a]
    for k in ("pvx", "pvy", "pvz"):
        o.arr(k)[sel] = rng.normal(0, 0.4, m)
    o.pflag[sel] = 5
    o.pAir[sel] = np.where(rng.random(m) < 0.2, 1.0, 0.0).astype(np.float32)
    fs = to_device(o)
    before = o.arr("pvx")[:nP].copy()
    o.stage("ice_contacts")
    fs.stage("ICE_CONTACTS")
    if kind in ("chain", "clump"):
        assert np.any(o.arr("pvx")[:nP] != before)
    assert np.array_equal(fs.pAir, o.pAir[:nP])
    for k in ("pvx", "pvy", "pvz"):
        assert np.array_equal(fs.download(k), o.arr(k)[:nP]), k
    fs.close()
