"""The tangent's assembly at the edges of its split: slices of one row and of
many, rows of one block, a ragged last group, particles numbered against
their positions, bonds damaged or broken on one side.  Every block against
the oracle's; a block is a sum of at most some 30 products of O(1) terms in
another order, so 1e-13 of the largest entry holds it."""
import numpy as np
import pytest

from lpm_cases import make_gpu, make_oracle, oracle, pkg
from test_gpu_onchip import CASES

capi = pkg.capi
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tangent", [capi.TANGENT_SYMMETRIC, capi.TANGENT_AS_WRITTEN])
@pytest.mark.parametrize("name", list(CASES))
def test_assembly_matches_the_oracle(name, tangent):
    case = CASES[name]()
    g, o = make_gpu(*case), make_oracle(*case)
    rng = np.random.default_rng(4)
    d = np.where(rng.random(g.nb) < 0.1, rng.random(g.nb), 0.0)
    d[rng.random(g.nb) < 0.03] = 1.0
    x = case[1] + 1e-3 * rng.standard_normal(case[1].shape) * (np.arange(3) < case[0])
    for s, key in ((g, capi.B_BDAMAGE), (o, oracle.BDAMAGE)):
        (s.upload if s is g else s.set_bond)(key, d)
    g.upload(capi.F_XYZ, x)
    o.set(oracle.XYZ, x)
    g.update()
    o.update()
    g.assemble(tangent, capi.BC_NONE)
    o.assemble(sym=1 if tangent == capi.TANGENT_SYMMETRIC else 0, bc=0)
    A, B = g.K_bsr(), o.K_bsr()
    err = np.abs(A - B).max()
    print("[assemble] %s: %.1e of %.1e" % (name, err, np.abs(B).max()))
    assert err <= 1e-13 * np.abs(B).max()
    g.close()
