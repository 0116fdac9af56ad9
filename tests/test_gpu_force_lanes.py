"""The force pass with one, two and four lanes to a particle (chosen by the
number of particles): a bond's values against the oracle bit for bit where
they are the reference's, sums to rounding.  Sizes on both sides of the
choices, particles with fewer bonds than lanes, broken bonds."""
import numpy as np
import pytest

from lpm_cases import cube, make_gpu, make_oracle, oracle, pkg, plate
from test_gpu_onchip import CASES

capi = pkg.capi
pytestmark = pytest.mark.gpu

# a particle's sum of at most 18 bonds: 18 roundings of the largest term and
# as many in the oracle's, held against the largest value of the field
TOL = 1e-13
SIZES = {"cube 3": CASES["cube 3"], "plate 4x3": CASES["plate 4x3"], "bar 2x3x11": CASES["bar 2x3x11"],
         "plate 81x101 (2 lanes)": lambda: plate(81, 101), "plate 60x61 (4 lanes)": lambda: plate(60, 61),
         "cube 20 (2 lanes)": lambda: cube(20), "cube 55 (1 lane)": lambda: cube(55)}


@pytest.mark.parametrize("name", list(SIZES))
def test_force_pass(name):
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
    assert np.array_equal(g.download(capi.B_DIS), o.get_bond(oracle.DIS))
    assert np.array_equal(g.download(capi.B_BSTRAIN), o.get_bond(oracle.BSTRAIN))
    for a, b in ((capi.F_PIN, oracle.PIN), (capi.F_STRESS, oracle.STRESS), (capi.F_DLE_TOT, oracle.DLE_TOT),
                 (capi.F_CS_SUM, oracle.CS_SUM), (capi.F_DVIS, oracle.DVIS)):
        u, v = np.ravel(g.download(a)), np.ravel(o.get(b))
        assert np.abs(u - v).max() <= TOL * max(np.abs(v).max(), 1.0), a
    g.close()
