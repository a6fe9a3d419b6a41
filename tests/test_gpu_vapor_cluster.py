"""The vapour pass at parcel counts around its blocks (512 parcels) and rounds
(4096 over the cluster): every draw of the two serial streams lands on the
reference's parcel, so the stream states and the flags match the oracle."""
import numpy as np
import pytest

from helpers import planet, to_device, PLAIN32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 511, 513, 4096, 4099, 8200])
def test_streams(count):
    o = planet("planet32", **PLAIN32)
    nP = o.nP
    rng = np.random.default_rng(count)
    sel = rng.choice(nP, min(count, nP), replace=False)
    n = len(sel)
    assert n == count
    c, R = o.nx * o.dx / 2, o.scalars.oceanR
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = R + rng.uniform(-0.1, 0.4, n)
    o.px[sel] = c + d[:, 0] * r; o.py[sel] = c + d[:, 1] * r; o.pz[sel] = c + d[:, 2] * r
    for a in (o.pvx, o.pvy, o.pvz):
        a[sel] = rng.normal(0, 0.5, n)
    o.pflag[sel] = rng.choice([2, 3], n)
    o.pT[sel] = rng.uniform(0.1, 0.5, n)
    o.pAir[sel] = rng.uniform(0, 1, n)
    fs = to_device(o)
    for _ in range(2):
        o.substep(0.01)
        fs._substep(0.01)
        so, sg = o.scalars, fs.scalars
        assert (sg.cfS, sg.bfS) == (so.cfS, so.bfS)
    assert np.array_equal(fs.pflag, o.pflag[:nP])
    for k in ("px", "py", "pz"):
        # parcels only: two substeps of double arithmetic rounded to float
        assert np.max(np.abs(fs.download(k)[sel].astype(np.float64) - o.arr(k)[sel])) <= 1e-5 * o.nx, k
    fs.close()
