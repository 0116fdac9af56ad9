"""The mixed solve with the stiffness scaled by powers of two.  Scaling it is
exact in every quantity of the solve as long as nothing leaves FP32's range: the
iterations are the same.  r.z and p.q go with the stiffness' inverse; where they
fall below the range the solve breaks down and runs again in FP64, to the same
tolerance."""
import pytest

from lpm_cases import cube, pkg, plate
from test_gpu_solve_paths import System

capi = pkg.capi
pytestmark = pytest.mark.gpu


def _scaled(case, k):
    dim, xyz, p1, p2, layer, Kn, Tv, cell = case
    return dim, xyz, p1, p2, layer, Kn * 2.0**k, Tv * 2.0**k, cell


@pytest.mark.parametrize("tol,exact", [(1e-10, 30), (1e-13, 20)])
@pytest.mark.parametrize("precond", [capi.PRECOND_JACOBI, capi.PRECOND_COARSE])
@pytest.mark.parametrize("make,size", [(plate, (40, 60)), (cube, (12,))])
def test_solve_of_scaled_stiffness(make, size, precond, tol, exact):
    out = {}
    for k in (0, -60, 10, 20, 30, 40, 50, 60, 70, 80, 90, 100):
        s = System(_scaled(make(*size), k), precond)
        s.g.upload(capi.F_RESIDUAL, s.b)
        s.g.reset_stats()
        it, rr, st = s.g.solve(capi.PREC_MIXED, tol)
        assert st == capi.OK and rr <= tol, k
        out[k] = (it, s.g.stats()["mixed_fallbacks"])
        s.g.close()
    print("[scale] tolerance %.0e: %s" % (tol, out))
    assert all(out[k] == out[0] for k in out if k <= exact) and out[0][1] == 0
