"""The bond force with one, two and four lanes to a particle, against the
oracle.  It has the owner's layer sum in it, so its last bits go with the lanes:
a sum of at most 18 terms, 18 roundings of the largest on either side, and a few
of the products: 1e-14 of the force's two terms at their largest.  The particles'
sums likewise, each against its own field's largest value."""
import numpy as np
import pytest

from lpm_cases import make_gpu, make_oracle, oracle, pkg
from test_gpu_force_lanes import SIZES

capi = pkg.capi
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(SIZES))
def test_bond_force(name):
    case = SIZES[name]()
    g, o = make_gpu(*case), make_oracle(*case)
    rng = np.random.default_rng(8)
    d = np.where(rng.random(g.nb) < 0.05, rng.random(g.nb), 0.0)
    d[rng.random(g.nb) < 0.02] = 1.0
    x = case[1] + 1e-3 * rng.standard_normal(case[1].shape) * (np.arange(3) < case[0])
    g.upload(capi.B_BDAMAGE, d)
    o.set_bond(oracle.BDAMAGE, d)
    g.upload(capi.F_XYZ, x)
    o.set(oracle.XYZ, x)
    g.update()
    o.update()
    assert np.array_equal(g.download(capi.B_DLE), o.get_bond(oracle.DLE))
    terms = 2 * np.abs(g.download(capi.B_KN)).max() * np.abs(o.get_bond(oracle.DLE)).max() + \
        2 * np.abs(g.download(capi.B_TV)).max() * 18 * np.abs(o.get_bond(oracle.DLE)).max()
    assert np.abs(g.download(capi.B_BFORCE) - o.get_bond(oracle.BFORCE)).max() <= 1e-14 * terms
    for a, b in ((capi.F_PIN, oracle.PIN), (capi.F_DLE_TOT, oracle.DLE_TOT), (capi.F_DVIS, oracle.DVIS)):
        u, v = np.ravel(g.download(a)), np.ravel(o.get(b))
        assert np.abs(u - v).max() <= 1e-13 * np.abs(v).max(), a
    g.close()
