"""The exact Jacobian's product with bonds damaged or broken on one side, whose
two directed bonds carry different weights, against central differences of the
oracle's internal force (as the undamaged states of test_gpu_adjoint: the
differences' error is some 1e-16 / 1e-6 of the force and 1e-12 of its third
derivative, held to 1e-6)."""
import numpy as np
import pytest

from lpm_cases import make_gpu, make_oracle, oracle, pkg
from test_gpu_adjoint import strained_state

capi = pkg.capi
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_jacobian_product_with_one_sided_damage(dim):
    args, x = strained_state(dim)
    g, o = make_gpu(*args), make_oracle(*args)
    rng = np.random.default_rng(12)
    d = np.where(rng.random(g.nb) < 0.2, rng.random(g.nb), 0.0)
    d[rng.random(g.nb) < 0.1] = 1.0
    g.upload(capi.B_BDAMAGE, d)
    o.set_bond(oracle.BDAMAGE, d)
    assert (d != d[g.bonds()["opp"]]).any()
    g.upload(capi.F_XYZ, x)
    g.update()
    n = len(x)
    v = rng.standard_normal(n * dim)
    Hv = g.apply_jacobian(v)

    def pin(xx):
        o.set(oracle.XYZ, xx)
        o.update()
        return o.get(oracle.PIN)[:, :dim].ravel().copy()

    V = np.zeros((n, 3))
    V[:, :dim] = v.reshape(n, dim)
    h = 1e-6
    fd = (pin(x + h * V) - pin(x - h * V)) / (2 * h)
    print("[jacobian] %d-D, one-sided damage: %.2e of the largest" % (dim, np.abs(Hv - fd).max() / np.abs(fd).max()))
    assert np.abs(Hv - fd).max() <= 1e-6 * np.abs(fd).max()
    g.close()
