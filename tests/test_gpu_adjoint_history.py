"""The backward step does not depend on what its handle did before: the same
state gives the same gradients, bit for bit, on a handle that has solved and on
one that has not.  Enough DOFs (92k) that the folds of its sums differ with the
number of blocks."""
import numpy as np
import pytest

from lpm_cases import cube, make_gpu, pkg

capi = pkg.capi
pytestmark = pytest.mark.gpu


def test_backward_step_of_a_fresh_handle():
    case = cube(32)
    xyz = case[1]
    x = xyz + 1e-4 * np.random.default_rng(5).standard_normal(xyz.shape)
    mask = np.zeros(xyz.shape, np.int32)
    mask[xyz[:, 2] < 1e-9] = 1
    c = np.random.default_rng(6).standard_normal(xyz.shape)
    out = []
    for solves in (False, True):
        g = make_gpu(*case)
        g.set_mask(mask)
        g.upload(capi.F_XYZ, x)
        g.update()
        if solves:
            g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
            g.upload(capi.F_RESIDUAL, c)
            assert g.solve(capi.PREC_MIXED, 1e-6)[2] == capi.OK
        out.append(g.backward_step(dJdpin=c, cg_tol=1e-8))
        g.close()
    assert out[0][2:] == out[1][2:]
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
